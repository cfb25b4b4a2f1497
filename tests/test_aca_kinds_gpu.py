"""The split of the ACA's blocks over quarter CTAs, CTAs and clusters: few long
blocks (no clusters), and one kind or several; the product of the compressed
operator against the dense one within its tolerance."""
import numpy as np
import pytest
import torch

from pyquake3d_gb300 import gf, mesh
from pyquake3d_gb300.hmatrix import HMatrix

pytestmark = pytest.mark.gpu
MU = 32038120320.0


@pytest.mark.parametrize("nx,nz,size", [(160, 6, 16), (100, 10, 16), (40, 10, 16), (30, 15, 32), (12, 6, 8)])
@pytest.mark.parametrize("half", [False, True])
def test_product_within_the_tolerance(cuda, nx, nz, size, half):
    nodes, tris = mesh.planar_fault(nx * 0.5, nz * 0.5, nx, nz)
    nodes = nodes.copy()
    nodes[:, 1] = 0.6 * nodes[:, 2]          # a dipping plane, below the surface
    nodes[:, 2] = 0.8 * nodes[:, 2]
    nodes[:, 2] -= nodes[:, 2].max() + 400.0
    H = HMatrix(nodes, tris, MU, MU, min_size=size, mini_leaf=size, halfspace=half, device=cuda, tol=1e-5)
    K, _ = gf.assemble_dense(nodes, tris, MU, MU, halfspace=half, fp32_copy=False, device=cuda)
    g = torch.Generator().manual_seed(nx)
    x = torch.randn((1, 2 * len(tris)), generator=g, dtype=torch.float64).to(cuda)
    ref = K @ x[0]
    assert float(torch.linalg.norm(H.apply(x)[0] - ref)) <= 1e-5 * float(torch.linalg.norm(ref))
