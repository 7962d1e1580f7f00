"""pb_masked_rows (filter, c2r, mask, r2c of a batch on the binned modes) against torch FFTs of the
same spectra: one-, two- and three-pass lengths, odd axes, radices 7, 11 and 13, whole, ragged and one-row
masks, one and three legs, maps in several chunks.

Tolerance: FP64 transforms of n points, error below 10 eps log2(n) of the largest output."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def grid_of(n, kf):
    from polybin3d_b200 import _native as nat
    g = nat.PBGrid()
    for i in range(3):
        g.n[i], g.kf[i] = n[i], kf[i]
    return g


def modes(n, kf):
    ka = [np.fft.fftshift(np.arange(-n[i] // 2, n[i] // 2)) * kf[i] for i in range(2)]
    kx, ky, kz = np.meshgrid(ka[0], ka[1], np.arange(n[2] // 2 + 1) * kf[2], indexing="ij")
    k = np.sqrt(kx ** 2 + ky ** 2 + kz ** 2)
    return k, np.divide(kz, k, out=np.zeros_like(k), where=k > 0)


def a_mask(kind, n, rng):
    m = np.zeros(n)
    if kind == "full":
        m = 0.5 + rng.random(n)
    elif kind == "row":
        m[n[0] // 2, n[1] - 1] = rng.random(n[2]) + 0.1
    else:  # a ragged corner with an empty plane and rows of either parity
        m[: n[0] // 2 + 1, : n[1] // 2 + 1] = rng.random((n[0] // 2 + 1, n[1] // 2 + 1, n[2]))
        m *= (rng.random(n[:2]) < 0.7)[..., None]
        m[1] = 0
        m[0, 0, 0] = 1.0
    return m


@pytest.mark.parametrize("kind", ["full", "ragged", "row"])
@pytest.mark.parametrize("n,kf,legs", [
    ((16, 12, 10), (1.0, 1.0, 1.0), 1),
    ((60, 72, 90), (1.0, 1.0, 1.0), 1),
    ((100, 64, 48), (1.0, 1.0, 1.0), 3),
    ((216, 15, 200), (0.1, 1.0, 0.1), 1),
    ((32, 48, 64), (1.0, 1.0, 1.0), 1),
    ((27, 35, 22), (1.0, 0.8, 1.2), 3),
    ((128, 20, 26), (1.0, 1.0, 1.0), 3),
    ((26, 162, 32), (1.0, 0.3, 1.0), 1),
    ((162, 18, 28), (0.2, 1.0, 1.0), 1),
    ((15, 22, 270), (1.0, 1.0, 0.1), 3),
    ((20, 13, 512), (1.0, 1.0, 0.05), 1),
])
def test_against_torch(n, kf, legs, kind):
    from polybin3d_b200 import _native as nat
    rng = np.random.default_rng(11)
    dev = torch.device("cuda")
    grid = grid_of(n, kf)
    k, mu = modes(n, kf)
    ny = min(np.asarray(n) // 2 * np.asarray(kf))
    edges = np.linspace(0.15 * ny, 0.97 * ny, 6)
    n_src, n_maps = 3, 40
    src = torch.fft.rfftn(torch.as_tensor(rng.standard_normal((n_src,) + n), device=dev), dim=(1, 2, 3))
    mask = torch.as_tensor(a_mask(kind, n, rng), device=dev)
    maps, want = [], []
    for m in range(n_maps):
        lg, f = [], 0
        for q in range(legs):
            b, s, l = int(rng.integers(0, 5)), int(rng.integers(0, n_src)), int(rng.choice([0, 2, 4]))
            lg.append((s, edges[b], edges[b + 1], l, 1.0 + q))
            w = {0: 1 + 0 * mu, 2: 1.5 * mu ** 2 - 0.5, 4: (35 * mu ** 4 - 30 * mu ** 2 + 3) / 8}[l]
            w = (1.0 + q) * w * ((edges[b] <= k) & (k < edges[b + 1]))
            f = f + src[s] * torch.as_tensor(w, device=dev)
        maps.append(lg)
        want.append(torch.fft.rfftn(mask * torch.fft.irfftn(f, s=n, norm="forward")))
    chain = nat.MaskedRows(grid, mask)
    k_out = float(edges[-1])
    out = torch.full((n_maps,) + tuple(want[0].shape), float("nan"), dtype=torch.complex128, device=dev)
    chain.run(src, maps, k_out, out, nat.Workspace(dev), src_stride=src[0].numel())
    sel = torch.as_tensor(k < k_out, device=dev)
    got, want = out[:, sel], torch.stack(want)[:, sel]
    assert bool(torch.isfinite(torch.view_as_real(got)).all())
    tol = 10 * np.finfo(np.float64).eps * np.log2(np.prod(n)) * float(want.abs().max())
    assert float((got - want).abs().max()) <= tol


def test_unsupported_length():
    from polybin3d_b200 import _native as nat
    with pytest.raises(NotImplementedError):
        nat.MaskedRows(grid_of((34, 32, 32), (1.0, 1.0, 1.0)), torch.ones(34, 32, 32, device="cuda", dtype=torch.float64))


@pytest.mark.parametrize("with_z", [True, False])
@pytest.mark.parametrize("n,kf", [((16, 12, 10), (1.0, 1.0, 1.0)), ((27, 35, 22), (1.0, 0.8, 1.2)),
                                  ((20, 13, 512), (1.0, 1.0, 0.05)), ((64, 9, 26), (1.0, 1.0, 1.0))])
def test_product_rows(n, kf, with_z):
    from polybin3d_b200 import _native as nat
    rng = np.random.default_rng(5)
    dev = torch.device("cuda")
    X, Z = (torch.as_tensor(rng.standard_normal((4,) + n), device=dev) for _ in range(2))
    pairs = [(int(i), int(j)) for i, j in rng.integers(0, 4, (37, 2))]
    grid = grid_of(n, kf)
    k, _ = modes(n, kf)
    k_out = 0.97 * min(np.asarray(n) // 2 * np.asarray(kf))
    want = torch.stack([torch.fft.rfftn(X[i] * X[j] - (Z[i] * Z[j] if with_z else 0)) for i, j in pairs])
    out = torch.full_like(want, float("nan"))
    nat.product_rows(grid, X, Z if with_z else None, pairs, k_out, out, nat.transform_table(grid, dev),
                     nat.Workspace(dev))
    sel = torch.as_tensor(k < k_out, device=dev)
    got, want = out[:, sel], want[:, sel]
    tol = 10 * np.finfo(np.float64).eps * np.log2(np.prod(n)) * float(want.abs().max())
    assert bool(torch.isfinite(torch.view_as_real(got)).all()) and float((got - want).abs().max()) <= tol
