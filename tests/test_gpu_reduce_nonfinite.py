"""Infinite and NaN modes in the folded k-bin reduction: every bin and product gets the infinity or NaN of the direct
sum over modes (numpy), the others stay as without them."""
import numpy as np
import pytest
import torch

from polybin3d_b200 import _native as nat

pytestmark = pytest.mark.gpu
LEG = {0: lambda m: 1.0 + 0 * m, 2: lambda m: 1.5 * m ** 2 - 0.5, 4: lambda m: (35 * m ** 4 - 30 * m ** 2 + 3) / 8}


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("mode", ["abs2", "cross"])
@pytest.mark.parametrize("ells", [[(0, 0)], [(0, 0), (2, 0)], [(0, 0), (2, 0), (4, 0)], [(2, 0)],
                                  [(0, 0), (0, 2), (2, 0), (2, 2)], [(a, b) for a in (0, 2, 4) for b in (0, 2, 4)]])
def test_infinite_modes(ells, mode, dtype):
    n, edges = (16, 15, 62), [0.5, 2.5, 4.0, 5.0, 6.0, 7.0]
    rng = np.random.default_rng(4)
    half = (n[0], n[1], n[2] // 2 + 1)
    x = torch.from_numpy(rng.standard_normal(half + (2,))).to(dtype)
    y = torch.from_numpy(rng.standard_normal(half + (2,)).__abs__()).to(dtype)
    x[1, 0, 0, 0] = float("inf")       # |k| = 1, on the plane kz = 0
    x[0, 0, 3, 1] = -float("inf")      # 3, along z
    x[14, 3, 3, 0] = float("inf")      # 4.7, between
    x[0, 5, 2, 0] = float("nan")       # 5.4
    g = nat.PBGrid()
    for i in range(3):
        g.n[i], g.kf[i] = n[i], 1.0
    out = torch.empty(1, len(ells), len(edges) - 1, dtype=torch.float64, device="cuda")
    prec = nat.precision_of(dtype)
    a, b, m = (x, None, nat.PB_RED_ABS2) if mode == "abs2" else (y, x, nat.PB_RED_CROSS)
    a, b = a.cuda(), b if b is None else b.cuda()
    nat.bin_reduce(g, prec, m, a, b, 1, edges, ells, 1.0, out, nat.Workspace(torch.device("cuda")))
    out = out.cpu().numpy()[0]
    ka = [np.fft.fftshift(np.arange(-n[i] // 2, n[i] // 2)) for i in range(2)]
    kx, ky, kz = np.meshgrid(ka[0], ka[1], np.arange(half[2]), indexing="ij")
    k = np.sqrt(kx ** 2.0 + ky ** 2 + kz ** 2)
    mu = np.divide(kz, k, out=np.zeros_like(k), where=k > 0)
    X, Y = x.double().numpy(), y.double().numpy()
    f = (1.0 + (kz > 0)) * ((X ** 2).sum(-1) if mode == "abs2" else (X * Y).sum(-1))
    for e, (la, lb) in enumerate(ells):
        for i in range(len(edges) - 1):
            sel = (edges[i] <= k) & (k < edges[i + 1])
            t = f[sel] * LEG[la](mu[sel]) * LEG[lb](mu[sel])
            want = np.sum(t)
            if np.isfinite(want):
                # as the finite reductions: 64 n eps of the sum of |terms|
                tol = 64 * t.size * np.finfo(np.float64).eps * np.sum(np.abs(f[sel]))
                assert abs(out[e, i] - want) <= tol, (e, i)
            else:
                assert np.array_equal([out[e, i]], [want], equal_nan=True), (e, i, out[e, i], want)


@pytest.mark.parametrize("ells", [[(4, 4), (2, 0), (0, 2), (4, 0)], [(2, 2), (4, 0), (0, 0)], [(4, 2), (2, 4)], [(4, 0)]])
def test_products_in_any_order(ells):
    """Orders and repeats of the products that share slots, on finite values."""
    n, edges = (10, 9, 12), [0.5, 2.5, 4.0]
    rng = np.random.default_rng(8)
    x = torch.from_numpy(rng.standard_normal((n[0], n[1], n[2] // 2 + 1, 2))).cuda()
    g = nat.PBGrid()
    for i in range(3):
        g.n[i], g.kf[i] = n[i], 1.0
    out = torch.empty(len(ells), 2, dtype=torch.float64, device="cuda")
    nat.bin_reduce(g, nat.PB_F64, nat.PB_RED_ABS2, x, None, 1, edges, ells, 1.0, out, nat.Workspace(torch.device("cuda")))
    ka = [np.fft.fftshift(np.arange(-n[i] // 2, n[i] // 2)) for i in range(2)]
    kx, ky, kz = np.meshgrid(ka[0], ka[1], np.arange(n[2] // 2 + 1), indexing="ij")
    k = np.sqrt(kx ** 2.0 + ky ** 2 + kz ** 2)
    mu = np.divide(kz, k, out=np.zeros_like(k), where=k > 0)
    f = (1.0 + (kz > 0)) * (x.cpu().numpy() ** 2).sum(-1)
    for e, (la, lb) in enumerate(ells):
        for i in range(2):
            sel = (edges[i] <= k) & (k < edges[i + 1])
            t = f[sel] * LEG[la](mu[sel]) * LEG[lb](mu[sel])
            assert abs(float(out[e, i]) - t.sum()) <= 64 * t.size * np.finfo(np.float64).eps * np.sum(f[sel])
