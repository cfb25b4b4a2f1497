"""The H-matrix keeps the source and receiver tables only (and the half-space
tables where it is one), not the dense assembly's workspace."""
import numpy as np
import pytest

from pyquake3d_gb300 import _lib


@pytest.mark.parametrize("N", [1, 7, 1000, 100001])
def test_sizes(N):
    L = _lib.load()
    full, half = L.pq3d_gf_setup_bytes(N, 0), L.pq3d_gf_setup_bytes(N, 1)
    assert full == 8 * N * (42 + 12) and half == full + 8 * N * (42 + 88)
    assert half < L.pq3d_gf_workspace_bytes(N)
    assert L.pq3d_gf_setup_bytes(0, 0) == L.pq3d_gf_setup_bytes(-3, 1) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("half", [False, True])
def test_hmatrix_holds_no_more(cuda, half):
    import torch

    from pyquake3d_gb300 import gf, mesh
    from pyquake3d_gb300.hmatrix import HMatrix
    mu = 32038120320.0
    nodes, tris = mesh.planar_fault(20.0, 10.0, 20, 10)
    nodes = nodes - np.array([0.0, 0.0, nodes[:, 2].max() + 500.0])
    H = HMatrix(nodes, tris, mu, mu, min_size=16, mini_leaf=16, halfspace=half, device=cuda)
    assert H.tables.numel() == _lib.load().pq3d_gf_setup_bytes(len(tris), int(half))
    K, _ = gf.assemble_dense(nodes, tris, mu, mu, halfspace=half, fp32_copy=False, device=cuda)
    x = torch.randn((1, 2 * len(tris)), generator=torch.Generator().manual_seed(1), dtype=torch.float64).to(cuda)
    ref = K @ x[0]
    assert float(torch.linalg.norm(H.apply(x)[0] - ref)) <= 1e-4 * float(torch.linalg.norm(ref))
