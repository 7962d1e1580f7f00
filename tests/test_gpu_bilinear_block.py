"""pb_bilinear_block_maps against sums in 64 bits: outputs that do not fill a block, voxel counts with and
without the 16-byte path, tile remainders, the largest number of maps, refilled coefficients."""
import numpy as np
import pytest
import torch

from polybin3d_b200 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n_g,n_out,n_vox", [(1, 1, 1), (3, 4, 64), (20, 5, 4099), (32, 33, 1000), (128, 7, 129)])
def test_bilinear_block(dtype, n_g, n_out, n_vox):
    rng = np.random.default_rng(n_g + n_out + n_vox)
    G = torch.from_numpy(rng.standard_normal((n_g, n_vox))).cuda().to(dtype)
    n_t = 6 * n_out
    o, i, j = rng.integers(0, n_out, n_t), rng.integers(0, n_g, n_t), rng.integers(0, n_g, n_t)
    plan = None
    for trial in range(2):
        c = rng.standard_normal(n_t)
        plan = nat.BilinearPlan(n_g, n_out, o, i, j, c, G.device) if plan is None else plan.with_coefficients(c)
        out = plan.maps(G).double()
        terms = torch.from_numpy(c).cuda()[:, None] * G.double()[i] * G.double()[j]
        at = torch.from_numpy(o).cuda()
        ref = torch.zeros(n_out, n_vox, dtype=torch.float64, device="cuda").index_add_(0, at, terms)
        size = torch.zeros_like(ref).index_add_(0, at, terms.abs())
        # n_t + 3 roundings at most on any term: its coefficient, two products and the sums
        bound = 1.01 * (n_t + 3) * (torch.finfo(dtype).eps / 2) * size
        if dtype == torch.float64:
            bound = 2 * bound   # the reference rounds as often
        assert bool(((out - ref).abs() <= bound).all())
    # a view of maps that does not start on 16 bytes
    if n_g > 1 and n_vox % 4:
        sub = nat.BilinearPlan(n_g - 1, n_out, o, i % (n_g - 1), j % (n_g - 1), c, G.device)
        assert torch.equal(sub.maps(G[1:]), sub.maps(G[1:].clone()))
