"""sum_m Y_lm(k) rfftn(Y_lm(r) a(r)) as one band-limited chain (products in the z transform, sum over m from
harmonics evaluated on the device), against the chain of whole grids; and the folded reduction of monopoles
about a line of sight that is not an axis."""
import contextlib
import io

import numpy as np
import pytest
import torch

from polybin3d_b200 import PolyBin3D
from polybin3d_b200 import _native as nat

pytestmark = pytest.mark.gpu


def box(n):
    with contextlib.redirect_stdout(io.StringIO()):
        return PolyBin3D([10.0 * n[0], 11.0 * n[1], 9.0 * n[2]], list(n), boxcenter=[900.0, 400.0, -700.0],
                         sightline="local", backend="cuda")


@pytest.mark.parametrize("l", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [(30, 27, 24), (48, 65, 60), (15, 45, 128)])
def test_band_limited_chain(n, l):
    b = box(n)
    a = torch.tensor(np.random.default_rng(l).standard_normal(n), device="cuda")
    kx, ky, kz = b.k_grids
    k = torch.as_tensor(np.sqrt(kx ** 2 + ky ** 2 + kz ** 2), device="cuda")
    k_out = 0.8 * float(np.min(b.kNy))
    whole = b.harmonics.apply_fourier(a, l)
    got = b.harmonics.apply_fourier(a, l, k_out=k_out)
    # two FP64 transforms of at most 2^17 points and 9 terms: below 200 roundings of the largest mode
    assert torch.all((got - whole)[k < k_out].abs() <= 200 * 2.0 ** -53 * whole.abs().max())
    assert torch.all(got[k >= k_out] == 0)


def test_length_without_a_chain_keeps_whole_grids():
    b = box((34, 24, 24))   # 34 = 2 x 17
    a = torch.tensor(np.random.default_rng(0).standard_normal((34, 24, 24)), device="cuda")
    assert torch.equal(b.harmonics.apply_fourier(a, 2, k_out=0.1), b.harmonics.apply_fourier(a, 2))


@pytest.mark.parametrize("n", [(8, 8, 8), (33, 20, 64)])
@pytest.mark.parametrize("mode", ["abs2", "cross"])
def test_monopole_about_a_line_of_sight(n, mode):
    rng = np.random.default_rng(3)
    half = (n[0], n[1], n[2] // 2 + 1)
    x, y = (torch.tensor(rng.standard_normal(half) + 1j * rng.standard_normal(half), device="cuda") for _ in range(2))
    edges = [0.05, 0.1, 0.13, 0.3, 0.45]
    out = []
    for los in (False, True):
        g = nat.PBGrid()
        for i, kf in enumerate((0.1, 0.05, 0.02)):
            g.n[i], g.kf[i] = n[i], kf
        if los:
            g.flags = 1
            for i, c in enumerate((0.6, 0.48, 0.64)):
                g.los[i] = c
        o = torch.empty(4, dtype=torch.float64, device="cuda")
        m, p, q = (nat.PB_RED_ABS2, x, None) if mode == "abs2" else (nat.PB_RED_CROSS, x, y)
        nat.bin_reduce(g, nat.PB_F64, m, p, q, 1, edges, [(0, 0)], 0.5, o, nat.Workspace(torch.device("cuda")))
        out.append(o)
    assert torch.equal(out[0], out[1])   # the monopole has no direction: the same sums in the same order
