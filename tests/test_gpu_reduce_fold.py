"""The folded k-bin reduction (few rows, global sightline, even Legendre orders) against the
direct FP64 sum over modes, on odd and even axes, one- to many-lane kz lines, edges that fall on
modes, empty and one-mode bins; membership is compared exactly through unit spectra.

Tolerance: sums of n terms (mu moments of either sign, coefficients up to 35/8 each) in FP64 against
numpy's: 64 n eps times the sum of |terms| without the Legendre weight is never reached by rounding."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
LEG = {0: lambda m: 1.0 + 0 * m, 2: lambda m: 1.5 * m ** 2 - 0.5, 4: lambda m: (35 * m ** 4 - 30 * m ** 2 + 3) / 8}


def geometry(n, kf):
    ka = [np.fft.fftshift(np.arange(-n[i] // 2, n[i] // 2)) * kf[i] for i in range(2)]
    kx, ky, kz = np.meshgrid(ka[0], ka[1], np.arange(n[2] // 2 + 1) * kf[2], indexing="ij")
    k = np.sqrt(kx ** 2 + ky ** 2 + kz ** 2)
    return k, np.divide(kz, k, out=np.zeros_like(k), where=k > 0), 1.0 + (kz > 0)


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("mode", ["abs2", "cross", "real2", "unit"])
@pytest.mark.parametrize("n,kf,edges,ells", [
    ((8, 8, 8), (1.0, 1.0, 1.0), [0.0, 1.0, 2.0, 3.0], [(0, 0), (2, 0)]),
    ((9, 7, 10), (0.3, 0.5, 0.4), [-1.0, 0.3, 0.30001, 0.9, 40.0], [(0, 0)]),
    ((16, 15, 62), (1.0, 1.0, 1.0), [2.5, 3.0, 5.0, 9.0, 9.5, 20.0], [(0, 0), (2, 0), (4, 0)]),
    ((33, 20, 64), (0.1, 0.2, 0.1), list(np.linspace(0.1, 2.0, 21)), [(0, 0), (0, 2), (2, 2), (4, 4), (2, 4)]),
    ((6, 40, 130), (1.0, 1.0, 1.0), list(np.linspace(1.0, 20.0, 65)), [(0, 0), (2, 0), (4, 0)]),
    ((1, 2, 2), (1.0, 1.0, 1.0), [0.5, 3.0], [(2, 0)]),
])
def test_fold_against_direct_sum(n, kf, edges, ells, mode, dtype):
    from polybin3d_b200 import _native as nat
    rng = np.random.default_rng(7)
    half = (n[0], n[1], n[2] // 2 + 1)
    rows = 3 if mode in ("abs2", "cross") else 1
    rt = np.float32 if dtype == "f32" else np.float64
    x = rng.standard_normal((rows,) + half + (2,)).astype(rt)
    y = rng.standard_normal(half + (2,)).astype(rt)
    k, mu, deg = geometry(n, kf)
    if mode == "abs2":
        f = (x.astype(np.float64) ** 2).sum(-1)
    elif mode == "cross":
        f = (x.astype(np.float64) * y.astype(np.float64)).sum(-1)
    elif mode == "real2":
        f = x[..., 0].astype(np.float64) ** 2
    else:
        f = np.ones((1,) + half)
    g = nat.PBGrid()
    for i in range(3):
        g.n[i], g.kf[i] = n[i], kf[i]
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")
    out = torch.empty(rows, len(ells), len(edges) - 1, dtype=torch.float64, device="cuda")
    prec = nat.PB_F32 if dtype == "f32" else nat.PB_F64
    m, a, b = {"abs2": (nat.PB_RED_ABS2, dev(x), None), "cross": (nat.PB_RED_CROSS, dev(y), dev(x)),
               "real2": (nat.PB_RED_REAL2, dev(x[0, ..., 0]), None), "unit": (nat.PB_RED_REAL2, None, None)}[mode]
    nat.bin_reduce(g, prec, m, a, b, rows, edges, ells, 0.5, out, nat.Workspace(torch.device("cuda")))
    out = out.cpu().numpy()
    eps = np.finfo(np.float64).eps
    for r in range(rows):
        for e, (la, lb) in enumerate(ells):
            for i in range(len(edges) - 1):
                sel = (edges[i] <= k) & (k < edges[i + 1])
                t = 0.5 * (deg * f[r])[sel]
                want = np.sum(t * LEG[la](mu[sel]) * LEG[lb](mu[sel]))
                assert abs(out[r, e, i] - want) <= 64 * max(1, t.size) * eps * np.sum(np.abs(t)), (r, e, i)
                if mode == "unit" and (la, lb) == (0, 0):
                    assert out[r, e, i] == want  # mode counts, exactly


@pytest.mark.parametrize("los", [False, True])
@pytest.mark.parametrize("rows,mode", [(16, "cross"), (33, "abs2"), (64, "cross"), (70, "cross")])
@pytest.mark.parametrize("n,kf,edges,ells", [
    ((8, 8, 8), (1.0, 1.0, 1.0), [0.0, 1.0, 2.0, 3.0], [(0, 0), (2, 0)]),
    ((9, 7, 10), (0.3, 0.5, 0.4), [-1.0, 0.3, 0.30001, 0.9, 40.0], [(0, 0)]),
    ((33, 20, 64), (0.1, 0.2, 0.1), list(np.linspace(0.1, 2.0, 21)), [(0, 0), (1, 0), (2, 0), (3, 2), (4, 4)]),
    ((6, 40, 130), (1.0, 1.0, 1.0), list(np.linspace(1.0, 20.0, 41)), [(0, 0), (2, 0), (4, 0)]),
    ((20, 12, 70), (1.0, 1.0, 1.0), list(np.linspace(1.0, 9.0, 65)), [(0, 0), (2, 0), (4, 0)]),
])
def test_many_rows_against_direct_sum(n, kf, edges, ells, rows, mode, los):
    """16 rows and more, FP64: the staged kernel (the last binning fits 32 rows a block only), odd
    orders and a tilted line of sight included; tolerance as above."""
    from polybin3d_b200 import _native as nat
    leg = dict(LEG)
    leg[1], leg[3] = lambda m: m, lambda m: 0.5 * m * (5 * m ** 2 - 3)
    rng = np.random.default_rng(3)
    half = (n[0], n[1], n[2] // 2 + 1)
    x = rng.standard_normal((rows,) + half + (2,))
    y = rng.standard_normal(half + (2,))
    k, mu, deg = geometry(n, kf)
    g = nat.PBGrid()
    for i in range(3):
        g.n[i], g.kf[i] = n[i], kf[i]
    if los:
        g.flags = nat.PB_GRID_LOS
        v = np.asarray([0.6, 0.0, 0.8])
        for i in range(3):
            g.los[i] = v[i]
        ka = [np.fft.fftshift(np.arange(-n[i] // 2, n[i] // 2)) * kf[i] for i in range(2)]
        kx, ky, kz = np.meshgrid(ka[0], ka[1], np.arange(n[2] // 2 + 1) * kf[2], indexing="ij")
        mu = np.divide(v[0] * kx + v[2] * kz, k, out=np.zeros_like(k), where=k > 0)
    f = (x ** 2).sum(-1) if mode == "abs2" else (x * y).sum(-1)
    dev = lambda t: torch.as_tensor(np.ascontiguousarray(t), device="cuda")
    out = torch.ones(rows, len(ells), len(edges) - 1, dtype=torch.float64, device="cuda")
    m, a, b = (nat.PB_RED_ABS2, dev(x), None) if mode == "abs2" else (nat.PB_RED_CROSS, dev(y), dev(x))
    nat.bin_reduce(g, nat.PB_F64, m, a, b, rows, edges, ells, 0.5, out, nat.Workspace(torch.device("cuda")),
                   accumulate=True)
    out = out.cpu().numpy() - 1.0
    eps = np.finfo(np.float64).eps
    for i in range(len(edges) - 1):
        sel = (edges[i] <= k) & (k < edges[i + 1])
        for e, (la, lb) in enumerate(ells):
            w = 0.5 * deg[sel] * leg[la](mu[sel]) * leg[lb](mu[sel])
            for r in range(rows):
                t = f[r][sel]
                tol = 64 * max(1, t.size) * eps * (1 + 0.5 * np.sum(deg[sel] * np.abs(t)))
                assert abs(out[r, e, i] - np.sum(w * t)) <= tol, (r, e, i)
