"""pb_shell_rows with mode lists around one step of 16 per block and around one step for every block (1,776 modes a
group of 64 columns and below), against sums in 64 bits.  Tolerance: FP64 sums of n products on both sides, below
2 n eps sum |terms|."""
import numpy as np
import pytest
import torch

from polybin3d_b200 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_modes", [0, 1, 15, 16, 17, 1776, 7103, 7105])
@pytest.mark.parametrize("rows,cols", [(1, 1), (9, 65), (32, 260)])
def test_parts(rows, cols, n_modes):
    grid = nat.PBGrid()
    for i, n in enumerate((16, 24, 40)):
        grid.n[i], grid.kf[i] = n, 1.0
    half = 16 * 24 * 21
    rng = np.random.default_rng(rows + n_modes)
    F = torch.as_tensor(rng.standard_normal((4, half, 2)), device="cuda")
    Q = torch.as_tensor(rng.standard_normal((cols, half, 2)), device="cuda")
    modes = torch.as_tensor(np.sort(rng.choice(half, n_modes, replace=False)).astype(np.int64), device="cuda")
    key = rng.integers(0, 4, rows).astype(np.int32)
    out = torch.full((rows, cols), 7.0, dtype=torch.float64, device="cuda")
    nat.shell_rows(grid, torch.view_as_complex(F), torch.view_as_complex(Q), modes, key, list(range(rows)), 1.0, out,
                   nat.Workspace("cuda"))
    deg = torch.where(modes % 21 > 0, 2.0, 1.0).double()
    a = (F[key][:, modes] * deg[:, None]).reshape(rows, -1)
    b = Q[:, modes].reshape(cols, -1)
    tol = 2 * n_modes * np.finfo(np.float64).eps * (a.abs() @ b.abs().T)
    assert bool(((out - a @ b.T).abs() <= tol).all())
