"""pb_shell_synth's harmonic weights (l1 = PB_HARMONIC + l^2 + m) against maps weighted by the
host's harmonic grids, with and without a weight grid, l = 1..4, all m.

Tolerance: the two form the same FP64 products in another order, 1e-12 of each map's largest value
(as the synthesis against its two-step form)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weight", [False, True])
@pytest.mark.parametrize("n,out_n,kf", [((32, 36, 40), (24, 30, 32), (0.01, 0.012, 0.009)),
                                        ((48, 48, 48), (48, 48, 48), (0.01, 0.01, 0.01))])
def test_against_host_grids(n, out_n, kf, weight):
    from polybin3d_b200 import _native as nat
    from polybin3d_b200.harmonics import real_harmonics
    dev = torch.device("cuda")
    g = nat.PBGrid()
    for i in range(3):
        g.n[i], g.kf[i] = n[i], kf[i]
    ka = [np.fft.fftshift(np.arange(-n[i] // 2, n[i] // 2)) * kf[i] for i in range(2)]
    kg = np.meshgrid(*ka, np.arange(n[2] // 2 + 1) * kf[2], indexing="ij")
    w = np.random.default_rng(1).random(kg[0].shape) + 0.5 if weight else np.ones(kg[0].shape)
    top = 0.8 * min(np.asarray(out_n) // 2 * np.asarray(kf))
    edges = [0.0, 0.4 * top, top]
    ws = nat.Workspace(dev)

    def maps(l1, grid):
        out = torch.empty((2,) + tuple(out_n), dtype=torch.float64, device=dev)
        specs = [(0, edges[i], edges[i + 1], l1, 0, 1.0, 1 if grid is not None else 0) for i in range(2)]
        nat.shell_synth(g, nat.PB_F64, None, out, specs, out_n, ws,
                        w=None if grid is None else torch.as_tensor(grid, device=dev))
        return out
    for l in range(1, 5):
        for m, y in enumerate(real_harmonics(kg, l)):
            got = maps(nat.PB_HARMONIC + l * l + m, w if weight else None)
            want = maps(0, w * y)
            assert float((got - want).abs().max()) <= 1e-12 * float(want.abs().max()), (l, m)


def test_bad_codes():
    from polybin3d_b200 import _native as nat
    dev = torch.device("cuda")
    g = nat.PBGrid()
    for i in range(3):
        g.n[i], g.kf[i] = 16, 1.0
    out = torch.empty((1, 16, 16, 16), dtype=torch.float64, device=dev)
    for l1, l2 in ((16, 0), (41, 0), (5, 0), (20, 2)):
        with pytest.raises(ValueError):
            nat.shell_synth(g, nat.PB_F64, None, out, [(0, 0.0, 5.0, l1, l2, 1.0, 0)], (16, 16, 16), nat.Workspace(dev))
