"""pb_shell_synth with each output length that has kernels of its own, three-pass lengths (320, 384, 512) and one that
takes the Stockham kernels (1250), on each axis in turn, against torch's inverse transform of the filtered spectrum in 64
bits; and tiled sets of three-pass and Stockham lengths against the plain maps.

Tolerance: a transform of n points in FP64 or FP32 (filter product rounded once, then three line transforms), error below
10 eps log2(n) of the map's largest value."""
import numpy as np
import pytest
import torch

from polybin3d_b200 import _native as nat

pytestmark = pytest.mark.gpu

LENGTHS = [48, 60, 64, 72, 80, 90, 96, 100, 108, 120, 128, 144, 150, 160, 180, 192, 200, 216, 240, 256, 320, 384, 512,
           1250]


def setup(n, f32_source):
    """Grid with the band at the same fraction of every axis, a spectrum, weights, four maps and their spectra."""
    rng = np.random.default_rng(n[0] + 3 * n[1] + 7 * n[2])
    g = nat.PBGrid()
    kf = [16.0 / m for m in n]
    for i in range(3):
        g.n[i], g.kf[i] = n[i], kf[i]
    src = torch.fft.rfftn(torch.as_tensor(rng.standard_normal((2,) + n), device="cuda"), dim=(1, 2, 3))
    if f32_source:
        src = src.to(torch.complex64)
    e = [0.9, 2.6, 4.4, 6.9]
    maps = [(0, e[0], e[1], 0, 0, 1.0, 0), (1, e[1], e[2], 2, 0, 2.0, 1), (0, e[2], e[3], 4, 2, 0.5, -1),
            (1, e[0], e[3], 0, 0, 1.0, 2)]
    k = [np.fft.fftfreq(n[i], 1.0 / n[i]) * kf[i] for i in (0, 1)] + [np.arange(n[2] // 2 + 1) * kf[2]]
    kx, ky, kz = (torch.as_tensor(t, device="cuda").reshape([-1 if i == j else 1 for j in range(3)])
                  for i, t in enumerate(k))
    mod = torch.sqrt(kx ** 2 + ky ** 2 + kz ** 2)
    mu2 = torch.where(mod > 0, kz / mod.clamp_min(1e-300), 0 * mod) ** 2
    w = (1 + 0.4 * torch.sin(3 * mod)).float()     # even in k, as every weight of a real field
    leg = {0: 1 + 0 * mu2, 2: 1.5 * mu2 - 0.5, 4: (35 * mu2 ** 2 - 30 * mu2 + 3) / 8}
    F = torch.stack([src[s].to(torch.complex128) * (leg[a] * leg[b] * c * w.double() ** p * ((mod >= lo) & (mod < hi)))
                     for s, lo, hi, a, b, c, p in maps])
    return g, src, w, maps, F


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("length", LENGTHS)
def test_length_on_axis(length, axis):
    n = tuple(length if i == axis else 16 for i in range(3))
    for prec, rd in ((nat.PB_F64, torch.float64), (nat.PB_F32, torch.float32), (nat.PB_F32_SRC_F64, torch.float32)):
        g, src, w, maps, F = setup(n, prec == nat.PB_F32)
        want = torch.fft.irfftn(F, s=n, dim=(1, 2, 3), norm="forward")
        out = torch.full(want.shape, float("nan"), dtype=rd, device="cuda")
        nat.shell_synth(g, prec, src, out, maps, n, nat.Workspace(out.device), w=w.to(rd))
        tol = 10 * torch.finfo(rd).eps * np.log2(np.prod(n)) * want.abs().amax((1, 2, 3))
        assert bool(((out.double() - want).abs().amax((1, 2, 3)) <= tol).all()), (prec, n)


@pytest.mark.parametrize("n", [(16, 16, 320), (16, 16, 512), (512, 16, 16), (16, 16, 1250), (1250, 18, 16)])
def test_tiled_set_equals_plain_maps(n):
    g, src, w, maps, _ = setup(n, False)
    ws = nat.Workspace(src.device)
    plain = torch.empty((len(maps),) + n, dtype=torch.float32, device="cuda")
    nat.shell_synth(g, nat.PB_F32_SRC_F64, src, plain, maps, n, ws, w=w)
    T = nat.TiledMaps(len(maps), 2, n, plain.device)
    nat.shell_synth(g, nat.PB_F32_SRC_F64, src, T, maps, n, ws, w=w)
    hi, lo = T.split_parts()
    assert torch.equal(T.factor_maps(), plain[:2])
    assert torch.equal(hi, plain.to(torch.bfloat16))
    assert torch.equal(lo, (plain - hi.float()).to(torch.bfloat16))
