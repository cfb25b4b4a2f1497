"""The H-matrix product of several right-hand sides: every run's result is bit
for bit that of the run alone, for every group width, with runs switched off,
leaves of more than one row pass and long rank rows (a CTA each)."""
import numpy as np
import pytest
import torch

from pyquake3d_gb300 import mesh
from pyquake3d_gb300.hmatrix import HMatrix

pytestmark = pytest.mark.gpu
MU = 32038120320.0


@pytest.fixture(scope="module", params=[(16, 32, 8192), (110, 32, 8192), (16, 16, 64)])
def hmat(request, cuda):
    min_size, mini_leaf, long_row = request.param
    nodes, tris = mesh.rough_fault(24.0, 12.0, 43, 20, seed=2, ratio=5e-3)
    old, HMatrix.LONG_ROW = HMatrix.LONG_ROW, long_row
    try:
        return HMatrix(nodes, tris[:1711], MU, MU, min_size=min_size, mini_leaf=mini_leaf, device=cuda)
    finally:
        HMatrix.LONG_ROW = old


@pytest.mark.parametrize("B", [2, 3, 4, 5, 7, 8, 9, 11, 16, 37])
def test_runs_match_the_run_alone(cuda, hmat, B):
    H = hmat
    g = torch.Generator().manual_seed(B)
    X = (torch.randn((B, 2 * H.N), generator=g, dtype=torch.float64) * 10.0 ** torch.randint(-9, 3, (B, 1), generator=g)
         ).to(cuda)
    alone = torch.cat([H.apply(X[r:r + 1]) for r in range(B)])
    assert torch.equal(H.apply(X), alone)
    # switched off: its row of the output is left as it was
    on = torch.as_tensor(np.random.default_rng(B).random(B) < 0.6).to(cuda)
    for active in (on, torch.zeros_like(on), on.logical_not()):
        out = torch.full_like(alone, -7.0)
        H.apply(X, out=out, active=active.to(torch.int32))
        assert torch.equal(out, torch.where(active[:, None], alone, -7.0))
