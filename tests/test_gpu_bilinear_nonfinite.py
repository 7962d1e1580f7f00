"""pb_bilinear_maps (one output at a time) against sums in 64 bits, and a NaN or an infinity of one map in the blocks of
four: it reaches the outputs that use the map, as in pb_bilinear_maps, and no other output of their block."""
import ctypes

import numpy as np
import pytest
import torch

from polybin3d_b200 import _native as nat

pytestmark = pytest.mark.gpu


def one_by_one(G, n_out, o, i, j, c):
    """pb_bilinear_plan and pb_bilinear_maps."""
    lib = nat.load()
    o, i, j = (np.ascontiguousarray(x, dtype=np.int32) for x in (o, i, j))
    c = np.ascontiguousarray(c, dtype=np.float64)
    size, n = ctypes.c_size_t(), np.zeros(1, dtype=np.int32)
    plan = (G.shape[0], n_out, nat.hptr(o), nat.hptr(i), nat.hptr(j), nat.hptr(c), len(o))
    nat.check(lib.pb_bilinear_plan(*plan, None, ctypes.byref(size), nat.hptr(n)))
    table = np.zeros(size.value, dtype=np.uint8)
    nat.check(lib.pb_bilinear_plan(*plan, nat.hptr(table), ctypes.byref(size), nat.hptr(n)))
    table = torch.from_numpy(table).cuda()
    out = torch.empty((n_out, G.shape[1]), dtype=G.dtype, device=G.device)
    nat.check(lib.pb_bilinear_maps(nat.precision_of(G.dtype), G.shape[1], nat.ptr(G), G.shape[0], nat.ptr(table), int(n[0]),
                                   n_out, nat.ptr(out), nat.stream_ptr()))
    return out


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n_g,n_out,n_vox", [(1, 1, 1), (20, 5, 4099), (128, 7, 1000)])
def test_one_output_at_a_time(n_g, n_out, n_vox, dtype):
    rng = np.random.default_rng(n_g + n_out + n_vox)
    G = torch.from_numpy(rng.standard_normal((n_g, n_vox))).cuda().to(dtype)
    n_t = 6 * n_out
    o, i, j = rng.integers(0, n_out, n_t), rng.integers(0, n_g, n_t), rng.integers(0, n_g, n_t)
    c = rng.standard_normal(n_t)
    out = one_by_one(G, n_out, o, i, j, c).double()
    terms = torch.from_numpy(c).cuda()[:, None] * G.double()[i] * G.double()[j]
    at = torch.from_numpy(o).cuda()
    ref = torch.zeros(n_out, n_vox, dtype=torch.float64, device="cuda").index_add_(0, at, terms)
    size = torch.zeros_like(ref).index_add_(0, at, terms.abs())
    # n_t + 3 roundings at most on any term, and as many of the reference
    assert bool(((out - ref).abs() <= 2.02 * (n_t + 3) * (torch.finfo(dtype).eps / 2) * size).all())


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n_g,n_out,n_vox", [(6, 7, 4096), (6, 7, 4099), (40, 9, 70_000)])
def test_only_outputs_that_use_the_map(n_g, n_out, n_vox, dtype):
    rng = np.random.default_rng(n_g + n_vox)
    G = torch.from_numpy(rng.standard_normal((n_g, n_vox))).cuda().to(dtype)
    n_t = 5 * n_out
    o, i, j = rng.integers(0, n_out, n_t), rng.integers(0, n_g, n_t), rng.integers(0, n_g, n_t)
    i[:3], j[:3] = [0, 1, 0], [2, 0, 0]           # map 0 as either factor and squared
    keep = (o < 2) | ((i != 0) & (j != 0))        # in the first outputs only
    o[:3] = [0, 1, 0]
    keep[:3] = True
    o, i, j = o[keep], i[keep], j[keep]
    c = rng.uniform(0.5, 1.5, len(o))
    plan = nat.BilinearPlan(n_g, n_out, o, i, j, c, G.device)
    clean = plan.maps(G)
    bad = {3: float("nan"), n_vox // 2: float("inf"), n_vox - 1: -float("inf")}
    for x, v in bad.items():
        G[0, x] = v
    got = plan.maps(G)
    uses = sorted({int(a) for a, p, q in zip(o, i, j) if p == 0 or q == 0})
    rest = [a for a in range(n_out) if a not in uses]
    at = torch.tensor(list(bad), device="cuda")
    assert uses == [0, 1]
    assert torch.equal(got[rest], clean[rest])
    assert not torch.isfinite(got[uses][:, at]).any()
    alone = one_by_one(G, n_out, o, i, j, c)
    assert torch.equal(torch.nan_to_num(got[uses][:, at], nan=7.0), torch.nan_to_num(alone[uses][:, at], nan=7.0))
    other = torch.ones(n_vox, dtype=torch.bool, device="cuda")
    other[at] = False
    # (the values beside a bad voxel are summed in the same order, with the zero coefficients left out)
    assert torch.equal(got[:, other], clean[:, other])
