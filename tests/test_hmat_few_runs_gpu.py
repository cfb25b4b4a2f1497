"""The H-matrix product of a batch at the sizes where its launch changes: run by
run or in groups (few leaves), half or whole row passes, and a batch of which one
run takes part (many leaves): every run's result has the bits of the run alone,
and the rows of the others stay as they were."""
import numpy as np
import pytest
import torch

from pyquake3d_gb300 import mesh
from pyquake3d_gb300.hmatrix import HMatrix

pytestmark = pytest.mark.gpu
MU = 32038120320.0


# (columns, rows, min_size, leaves at least, at most)
@pytest.fixture(scope="module", params=[(40, 20, 64, 24, 40), (70, 35, 64, 120, 136), (120, 30, 5, 1200, 4000)])
def hmat(request, cuda):
    nx, nz, size, lo, hi = request.param
    nodes, tris = mesh.rough_fault(nx * 0.5, nz * 0.5, nx, nz, seed=3, ratio=5e-3)
    H = HMatrix(nodes, tris, MU, MU, min_size=size, mini_leaf=size, device=cuda)
    assert lo <= len(H.leaves_host) <= hi
    return H


@pytest.mark.parametrize("B", [2, 3, 8, 9, 10, 16, 24])
def test_few_runs_match_the_run_alone(cuda, hmat, B):
    H = hmat
    g = torch.Generator().manual_seed(B)
    X = torch.randn((B, 2 * H.N), generator=g, dtype=torch.float64).to(cuda)
    alone = torch.cat([H.apply(X[r:r + 1]) for r in range(B)])
    assert torch.equal(H.apply(X), alone)
    rng = np.random.default_rng(B)
    masks = [np.arange(B) == r for r in (0, B // 2, B - 1)] + [np.arange(B) < 2, np.arange(B) != 1, rng.random(B) < 0.5,
                                                               np.zeros(B, bool), np.ones(B, bool)]
    for m in masks:
        on = torch.as_tensor(m).to(cuda)
        out = torch.full_like(alone, -7.0)
        H.apply(X, out=out, active=on.to(torch.int32))
        assert torch.equal(out, torch.where(on[:, None], alone, -7.0)), m
