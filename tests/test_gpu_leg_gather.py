"""pb_leg_gather (legs of the bispectrum gradient: forward transform, shell filter and sum in one chain) against
whole transforms and the accumulating filter, over lengths of one, two and three passes, run-time and compile-time
plans, unequal axes, shells that touch, coincide and overlap, and two destinations."""
import numpy as np
import pytest
import torch

from polybin3d_b200 import _native as nat

pytestmark = pytest.mark.gpu


def grid(n, los):
    g = nat.PBGrid()
    for i, kf in enumerate((0.010, 0.013, 0.009)):
        g.n[i], g.kf[i] = n[i], kf
    if los:
        g.flags = 1
        for i, c in enumerate((0.6, 0.48, 0.64)):
            g.los[i] = c
    return g


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("m,n,los", [
    ((12, 16, 10), (12, 16, 10), False),     # one pass per axis
    ((48, 40, 64), (60, 64, 96), False),     # two passes; 40 has the run-time plan
    ((20, 18, 30), (33, 21, 50), True),      # odd data axes, a line of sight that is no axis
    ((320, 24, 20), (320, 24, 20), False),   # three passes along x
    ((20, 24, 320), (20, 30, 320), False),   # ... and along z
])
def test_against_filter_of_whole_transforms(m, n, los, dtype):
    rng = np.random.default_rng(m[0] + n[2])
    kf = (0.010, 0.013, 0.009)
    top = 0.98 * min((min(m[i], n[i]) // 2 - 2) * kf[i] for i in range(3))
    e = [0.3 * top, 0.55 * top, 0.8 * top, top]
    legs = [(e[0], e[1], 0, 1.0, 0), (e[1], e[2], 0, 1.0, 0), (e[2], e[3], 2, 0.5, 0), (e[0], e[1], 2, 2.0, 0),
            (e[1], e[2], 4, 1.0, 1)]
    for case in (legs, legs + [(-1.0, e[2], 0, 1.0, 1)]):      # the last shell overlaps the others
        R = torch.tensor(rng.standard_normal((len(case),) + m), dtype=dtype, device="cuda")
        cd = torch.complex128 if dtype == torch.float64 else torch.complex64
        half = (n[0], n[1], n[2] // 2 + 1)
        start = torch.tensor(rng.standard_normal((2,) + half + (2,)), device="cuda")
        got = torch.view_as_complex(start.clone()).to(cd)
        want = torch.view_as_complex(start.clone()).to(torch.complex128)
        nat.leg_gather(grid(n, los), R, case, got, nat.Workspace(R.device))
        k = [np.fft.fftfreq(n[i], 1.0 / n[i]) * kf[i] for i in (0, 1)] + [np.arange(half[2]) * kf[2]]
        kx, ky, kz = np.meshgrid(*k, indexing="ij")
        mod = np.sqrt(kx ** 2 + ky ** 2 + kz ** 2)
        mu = (0.6 * kx + 0.48 * ky + 0.64 * kz if los else kz) / np.where(mod > 0, mod, 1.0)
        leg = {0: 1.0 + 0 * mu, 2: 1.5 * mu ** 2 - 0.5, 4: (35 * mu ** 4 - 30 * mu ** 2 + 3) / 8}
        # the modes of the data grid on the map grid
        at = [torch.as_tensor(np.rint(k[i] / kf[i]).astype(np.int64) % m[i], device="cuda") for i in (0, 1)]
        size = 0.0
        for q, (lo, hi, l, scale, dst) in enumerate(case):
            F = torch.fft.rfftn(R[q].double())
            F = torch.nn.functional.pad(F, (0, max(0, half[2] - F.shape[2])))[:, :, :half[2]]
            w = torch.as_tensor(scale * leg[l] * ((mod >= lo) & (mod < hi)), device="cuda")
            want[dst] += F[at[0]][:, at[1]] * w
            size = max(size, float(F.abs().max()))
        # three transforms of at most 9 radix-2 levels each, filter and sums: below 100 roundings of the largest mode
        eps = 2.0 ** -53 if dtype == torch.float64 else 2.0 ** -24
        assert float((got - want).abs().max()) <= 100 * eps * size * 2.0


def test_refused_bands_and_lengths():
    R = torch.zeros((1, 12, 12, 12), dtype=torch.float64, device="cuda")
    ws = nat.Workspace(R.device)
    grad = torch.zeros((1, 12, 12, 7), dtype=torch.complex128, device="cuda")
    with pytest.raises(NotImplementedError):    # reaches the Nyquist frequency
        nat.leg_gather(grid((12, 12, 12), False), R, [(0.0, 0.08, 0, 1.0, 0)], grad, ws)
    with pytest.raises(NotImplementedError):    # 14 = 2 x 7: no map grid of the synthesis
        nat.leg_gather(grid((14, 14, 14), False), torch.zeros((1, 14, 14, 14), dtype=torch.float64, device="cuda"),
                       [(0.0, 0.02, 0, 1.0, 0)], torch.zeros((1, 14, 14, 8), dtype=torch.complex128, device="cuda"), ws)
    assert not grad.any()
