"""The spatial order of the assembly's tiles (meshes whose own order leaves
many edges per tile, calls of many pairs): the operator's bits do not depend on
which triangles share a tile, so a shuffled mesh gives the bits of its row
ranges, which are too small for the order, and of the mesh in its own order."""
import numpy as np
import pytest
import torch

from pyquake3d_gb300 import gf, mesh

pytestmark = pytest.mark.gpu
MU = 32038120320.0


@pytest.mark.parametrize("half,N", [(False, 4097), (False, 5001), (True, 1024), (True, 1111)])
@pytest.mark.parametrize("order", ["mesh", "shuffled"])
def test_bits_do_not_depend_on_the_order(cuda, half, N, order):
    nodes, tris = mesh.rough_fault(50.0, 51.0, 50, 51, seed=N, ratio=5e-3)
    if half:
        nodes = nodes - np.array([0.0, 0.0, nodes[:, 2].max() + 500.0])
    tris = np.ascontiguousarray(tris[:N])
    p = np.arange(N) if order == "mesh" else np.random.default_rng(N).permutation(N)
    K, K32 = gf.assemble_dense(nodes, tris[p], MU, MU, halfspace=half, device=cuda)
    for r0, r1 in ((0, 33), (N - 20, N)):
        part, part32 = gf.assemble_dense(nodes, tris[p], MU, MU, halfspace=half, device=cuda, rows=(r0, r1))
        assert torch.equal(part, K[3 * r0:3 * r1]) and torch.equal(part32, K32[3 * r0:3 * r1])
    if order == "shuffled":
        Km, _ = gf.assemble_dense(nodes, tris, MU, MU, halfspace=half, device=cuda)
        q = torch.as_tensor(p, device=cuda)
        assert torch.equal(K.view(N, 3, N, 2), Km.view(N, 3, N, 2)[q][:, :, q])
