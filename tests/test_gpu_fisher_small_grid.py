"""Fisher matrices on grids of 16 points an axis and below (whole transforms) against the band-limited chains on the same
realisations.  Both are a few FP64 transforms of some thousand points and sums over them: 1e-12 of the largest element."""
import contextlib
import io

import numpy as np
import pytest
import torch

import polybin3d_b200 as pb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["pk", "bk"])
@pytest.mark.parametrize("n", [(16, 16, 16), (16, 14, 12)])
def test_both_routes(n, kind, monkeypatch):
    mask = np.random.default_rng(1).uniform(0.0, 1.0, n)
    mask[n[0] // 2] = 0.0
    out = []
    for whole in (True, False):
        monkeypatch.setattr(pb.PolyBin3D, "one_pass_axes", whole)
        with contextlib.redirect_stdout(io.StringIO()):
            b = pb.PolyBin3D([10.0 * m for m in n], n)
            edges = np.linspace(float(b.kF.max()), 0.6 * float(b.kNy.min()), 4)
            est = pb.PSpec(b, edges, lmax=2, mask=mask) if kind == "pk" else pb.BSpec(b, edges, lmax=2, mask=mask)
            F = est.compute_fisher(2, noise="philox")
        assert (est._pointing().rows() is None) == whole
        out.append(torch.as_tensor(F).cpu().numpy())
    assert np.abs(out[0] - out[1]).max() <= 1e-12 * np.abs(out[1]).max()
