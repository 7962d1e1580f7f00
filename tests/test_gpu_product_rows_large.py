"""pb_product_rows on a grid whose row blocks (65,536) are more than a launch takes in y, against torch's transform.
Tolerance as for the small grids: FP64 transforms of n points, error below 10 eps log2(n) of the largest output."""
import numpy as np
import pytest
import torch

from polybin3d_b200 import _native as nat

pytestmark = pytest.mark.gpu


def test_more_rows_than_grid_y():
    n, k_out = (512, 512, 500), 6.5
    g = nat.PBGrid()
    for i in range(3):
        g.n[i], g.kf[i] = n[i], 1.0
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(2)
    X = torch.randn((1,) + n, generator=gen, dtype=torch.float64, device=dev)
    out = torch.full((1, n[0], n[1], n[2] // 2 + 1), float("nan"), dtype=torch.complex128, device=dev)
    nat.product_rows(g, X, None, [(0, 0)], k_out, out, nat.transform_table(g, dev), nat.Workspace(dev))
    want = torch.fft.rfftn(X[0] * X[0])
    i = torch.arange(n[0], device=dev)
    f2 = torch.where(i < n[0] // 2, i, i - n[0]).double() ** 2
    sel = (f2[:, None, None] + f2[None, :, None] + torch.arange(n[2] // 2 + 1, device=dev).double() ** 2) < k_out ** 2
    got, want = out[0][sel], want[sel]
    tol = 10 * np.finfo(np.float64).eps * np.log2(np.prod(n)) * float(want.abs().max())
    assert bool(torch.isfinite(torch.view_as_real(got)).all()) and float((got - want).abs().max()) <= tol
