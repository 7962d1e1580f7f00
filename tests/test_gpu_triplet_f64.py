"""FP64 triplet contraction (matrix-instruction kernel) at the edges of its tiles: 8 pairs, 8 C maps, 128 or 64
voxels, 256 pairs and 32 C maps per block."""
import numpy as np
import pytest
import torch

from polybin3d_b200 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_a,n_b,n_c,n_trip,n_vox,shared", [
    (1, 1, 1, 1, 1, False),
    (2, 4, 8, 17, 127, False),          # one pair tile, one C tile; a ragged, unaligned voxel tile
    (3, 3, 9, 40, 128, False),          # 9 pairs, 9 C maps: one of each past a tile
    (16, 17, 33, 2000, 4097, False),   # 272 pairs and 33 C maps: a second group of both, odd rows (4-byte copies)
    (12, 12, 12, 150, 30_000, True),   # one set of maps
    (20, 5, 24, 300, 100_002, False),
])
def test_f64_contraction(n_a, n_b, n_c, n_trip, n_vox, shared):
    rng = np.random.default_rng(n_vox)
    A = torch.tensor(rng.standard_normal((n_a, n_vox)), device="cuda")
    B, C = (A, A) if shared else (torch.tensor(rng.standard_normal((n, n_vox)), device="cuda") for n in (n_b, n_c))
    every = np.stack(np.meshgrid(np.arange(n_a), np.arange(n_b), np.arange(n_c), indexing="ij"), -1).reshape(-1, 3)
    if n_a * n_b > 256:
        # every pair at least once
        first = every.reshape(-1, n_c, 3)[np.arange(n_a * n_b), rng.integers(0, n_c, n_a * n_b)]
        idx = np.unique(np.concatenate([first, rng.permutation(every)[:n_trip]]), axis=0)
    else:
        idx = rng.permutation(every)[:n_trip]
    idx = np.ascontiguousarray(rng.permutation(idx), dtype=np.int32)
    plan = nat.TripletPlan(n_a, n_b, n_c, idx, A.device)
    ws = nat.Workspace(A.device)
    out = torch.full((len(idx),), float("nan"), dtype=torch.float64, device="cuda")
    plan.contract(A, B, C, out, ws, method=nat.PB_TRIPLET_SIMT, scale=0.5)
    i = torch.as_tensor(idx, device="cuda", dtype=torch.long)
    for t0 in range(0, len(idx), 256):
        t = i[t0:t0 + 256]
        terms = A[t[:, 0]] * B[t[:, 1]] * C[t[:, 2]]
        # a term's two roundings and at most 256 voxels per block, 8 warps and 44 blocks in a chain,
        # as many again for the reference: fewer than 700 roundings, each of at most the sum of moduli
        bound = 0.5 * 700 * 2.0 ** -53 * terms.abs().sum(1)
        assert torch.all((out[t0:t0 + 256] - 0.5 * terms.sum(1)).abs() <= bound)


def test_f64_non_finite_stays_in_its_triplets():
    n_vox = 1000
    A = torch.ones((4, n_vox), dtype=torch.float64, device="cuda")
    C = torch.ones((9, n_vox), dtype=torch.float64, device="cuda")
    C[3, 17] = float("inf")
    C[8, 999] = float("nan")
    idx = np.asarray([(a, b, c) for a in range(4) for b in range(a, 4) for c in range(9)], dtype=np.int32)
    plan = nat.TripletPlan(4, 4, 9, idx, A.device)
    out = torch.empty(len(idx), dtype=torch.float64, device="cuda")
    plan.contract(A, A, C, out, nat.Workspace(A.device), method=nat.PB_TRIPLET_SIMT)
    got = out.cpu().numpy()
    assert np.all(np.isposinf(got[idx[:, 2] == 3])) and np.all(np.isnan(got[idx[:, 2] == 8]))
    assert np.all(got[(idx[:, 2] != 3) & (idx[:, 2] != 8)] == n_vox)
