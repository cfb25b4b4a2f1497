"""Assembly into mapped host memory (which keeps the mesh's own order in full
space) of meshes whose device assembly orders its tiles anew: the device
operator's bits, both precisions."""
import numpy as np
import pytest
import torch

from pyquake3d_gb300 import gf, mesh

pytestmark = pytest.mark.gpu
MU = 32038120320.0


@pytest.mark.parametrize("half,N", [(False, 4097), (True, 1025)])
@pytest.mark.parametrize("order", ["mesh", "shuffled"])
def test_host_output_has_the_bits_of_the_device_output(cuda, half, N, order):
    nodes, tris = mesh.rough_fault(50.0, 51.0, 50, 51, seed=N, ratio=5e-3)
    if half:
        nodes = nodes - np.array([0.0, 0.0, nodes[:, 2].max() + 500.0])
    tris = np.ascontiguousarray(tris[:N])
    if order == "shuffled":
        tris = np.ascontiguousarray(tris[np.random.default_rng(N).permutation(N)])
    K, K32 = gf.assemble_dense(nodes, tris, MU, MU, halfspace=half, device=cuda)
    H = torch.full((3 * N, 2 * N), float("nan"), dtype=torch.float64).pin_memory()
    H32 = torch.full((3 * N, 2 * N), float("nan"), dtype=torch.float32).pin_memory()
    gf.assemble_dense_host(nodes, tris, MU, MU, halfspace=half, fp32_copy=True, out64=H, out32=H32)
    assert torch.equal(H, K.cpu()) and torch.equal(H32, K32.cpu())
