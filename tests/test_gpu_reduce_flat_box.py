"""The staged k-bin reduction (16 rows and more, FP64) on boxes much longer in z than in x and y, with bins that start
where kz = 0 modes begin: unit spectra, so every bin is its mode count, exactly."""
import numpy as np
import pytest
import torch

from polybin3d_b200 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kf,lo", [((1.0, 1.0, 1.0), 3.0),
                                   ((1.0535579060570495, 0.9951035422927954, 0.001), 8.733322828531696),
                                   ((3.010273803286439, 2.798354724447148, 0.001), 21.256915366789535),
                                   ((20.841333724541542, 20.16275678722861, 0.001), 111.73708764845432)])
def test_mode_counts(kf, lo):
    n, rows = (16, 16, 64), 16
    edges = [lo, 1.2 * lo, 1.5 * lo]
    ka = [np.fft.fftshift(np.arange(-n[i] // 2, n[i] // 2)) * kf[i] for i in range(2)]
    kx, ky, kz = np.meshgrid(ka[0], ka[1], np.arange(n[2] // 2 + 1) * kf[2], indexing="ij")
    k = np.sqrt(kx ** 2 + ky ** 2 + kz ** 2)
    deg = 1.0 + (kz > 0)
    want = [deg[(edges[i] <= k) & (k < edges[i + 1])].sum() for i in range(2)]
    g = nat.PBGrid()
    for i in range(3):
        g.n[i], g.kf[i] = n[i], kf[i]
    x = torch.ones((rows,) + k.shape, dtype=torch.complex128, device="cuda")
    out = torch.empty(rows, 1, 2, dtype=torch.float64, device="cuda")
    nat.bin_reduce(g, nat.PB_F64, nat.PB_RED_ABS2, x, None, rows, edges, [(0, 0)], 1.0, out,
                   nat.Workspace(torch.device("cuda")))
    assert np.array_equal(out.cpu().numpy()[:, 0], np.broadcast_to(want, (rows, 2)))
