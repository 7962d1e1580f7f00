"""Bispectrum gradient on map grids with odd axes (synthesis='cufft': the bands leave no smaller even grid) against
torch's autograd of the same sums in 64 bits.  Both sides make a few FP64 transforms of 4,800 points and sums over
them: 1e-12 of the largest component leaves two orders of margin."""
import contextlib
import io

import numpy as np
import pytest
import torch

import polybin3d_b200 as pb
from polybin3d_b200.autograd import bk_numerator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(15, 20, 16), (15, 21, 16)])
def test_odd_map_grid(n):
    with contextlib.redirect_stdout(io.StringIO()):
        b = pb.PolyBin3D([100.0 * m for m in n], n)
        kf = float(b.kF.max())
        edges = np.linspace(kf, 0.9 * float(b.kNy.min()), 4)
        bs = pb.BSpec(b, edges, lmax=2, synthesis="cufft")
        bs._compute_symmetry_factor()
    assert bs.map_grid[0] == 15
    gen = torch.Generator(device=b.device).manual_seed(5)
    d = torch.randn(n, generator=gen, dtype=torch.float64, device=b.device)
    v = torch.randn(bs.N_bins, generator=gen, dtype=torch.float64, device=b.device)
    x = d.clone().requires_grad_(True)
    num = bk_numerator(bs, x)
    (grad,) = torch.autograd.grad(num, x, grad_outputs=v)
    k = torch.as_tensor(b.modk_grid, device=b.device)
    kz = torch.arange(n[2] // 2 + 1, device=b.device).double() * float(b.kF[2])
    mu2 = torch.where(k > 0, kz / k.clamp_min(1e-300), 0 * k) ** 2
    leg = {0: 1 + 0 * mu2, 2: 1.5 * mu2 - 0.5}
    y = d.clone().requires_grad_(True)
    X = torch.fft.rfftn(y)
    g = {(l, i): torch.fft.irfftn(X * leg[l] * ((k >= edges[i]) & (k < edges[i + 1])), s=n) for l in (0, 2)
         for i in range(3)}
    want = torch.stack([(g[0, i] * g[0, j] * g[l, q]).sum() for i, j, q, l in bs.all_bins.tolist()])
    want = want * (b.volume / b.nreal) / torch.as_tensor(bs.sym_factor, device=b.device)
    (gw,) = torch.autograd.grad(want, y, grad_outputs=v)
    assert float((num - want).detach().abs().max()) <= 1e-12 * float(want.detach().abs().max())
    assert float((grad - gw).abs().max()) <= 1e-12 * float(gw.abs().max())
