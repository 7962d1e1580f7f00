"""The finalize passes of the reductions (columns summed by 32 x 16 thread blocks): counts at
the edges of a block, one to many partials per column.

Tolerance: FP64 sums of n terms of either sign against torch's, error below n eps sum |terms|."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_vox", [100, 2048, 17 * 128 + 5, 600 * 128])
@pytest.mark.parametrize("n_trip", [1, 31, 32, 33, 64])
def test_triplet_sums(n_trip, n_vox):
    from polybin3d_b200 import _native as nat
    rng = np.random.default_rng(n_trip + n_vox)
    G = torch.as_tensor(rng.standard_normal((5, n_vox)), device="cuda")
    every = [(a, b, c) for a in range(5) for b in range(5) for c in range(5)]
    idx = np.asarray([every[i] for i in rng.choice(len(every), n_trip, replace=False)], dtype=np.int32)
    plan = nat.TripletPlan(5, 5, 5, idx, "cuda")
    out = torch.empty(n_trip, dtype=torch.float64, device="cuda")
    plan.contract(G, G, G, out, nat.Workspace("cuda"))
    terms = G[idx[:, 0]] * G[idx[:, 1]] * G[idx[:, 2]]
    tol = n_vox * np.finfo(np.float64).eps * terms.abs().sum(1)
    assert bool(((out - terms.sum(1)).abs() <= tol).all())


@pytest.mark.parametrize("n_modes", [1, 31, 32, 33, 4000])
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 31), (32, 33)])
def test_shell_rows(rows, cols, n_modes):
    from polybin3d_b200 import _native as nat
    grid = nat.PBGrid()
    for i, n in enumerate((16, 18, 40)):
        grid.n[i], grid.kf[i] = n, 1.0
    half = 16 * 18 * 21
    rng = np.random.default_rng(rows + cols + n_modes)
    F = torch.as_tensor(rng.standard_normal((4, half, 2)), device="cuda")
    Q = torch.as_tensor(rng.standard_normal((cols, half, 2)), device="cuda")
    modes = torch.as_tensor(np.sort(rng.choice(half, n_modes, replace=False)).astype(np.int64), device="cuda")
    key = rng.integers(0, 4, rows).astype(np.int32)
    out = torch.zeros(rows, cols, dtype=torch.float64, device="cuda")
    nat.shell_rows(grid, torch.view_as_complex(F), torch.view_as_complex(Q), modes, key, list(range(rows)), 0.5, out,
                   nat.Workspace("cuda"))
    deg = torch.where(modes % 21 > 0, 2.0, 1.0)
    terms = 0.5 * (F[key][:, modes] * deg[:, None]).reshape(rows, 1, -1) * Q[:, modes].reshape(1, cols, -1)
    tol = 2 * n_modes * np.finfo(np.float64).eps * terms.abs().sum(2)
    assert bool(((out - terms.sum(2)).abs() <= tol).all())
