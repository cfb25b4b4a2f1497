"""The dense stepper at the sizes where its launch changes (warps per receiver,
four lanes per cell, cells per block) against the batched FP64 stepper, which
evaluates the reference formula with a thread per cell: states and slips to
the project's 1e-9 after the same accepted steps, pore pressure on and off."""
import numpy as np
import pytest
import torch

from pyquake3d_gb300 import gf, mesh
from pyquake3d_gb300.ensemble import Ensemble
from pyquake3d_gb300.QDsim_gpu import DenseDeviceSim, initial_state

pytestmark = pytest.mark.gpu
MU, CS = 32038120320.0, 3464.0


def _case(N, cuda):
    nz = max(1, int(np.sqrt(N / 4)))
    nx = -(-N // (2 * nz))
    nodes, tris = mesh.rough_fault(nx * 1.0, nz * 1.0, nx, nz, seed=N, ratio=2e-3) if nx > 1 and nz > 1 else \
        mesh.planar_fault(nx * 1.0, nz * 1.0, nx, nz)
    tris = np.ascontiguousarray(tris[:N])
    _, xg = mesh.element_frames(nodes, tris)
    K64, K32 = gf.assemble_dense(nodes, tris, MU, MU, device=cuda)
    return K64, K32, mesh.friction_table(xg, nx * 1e3, nz * 1e3, seed=1)


@pytest.mark.parametrize("N", [1, 2, 33, 303, 305, 607, 609, 1215, 1217, 2431, 2433, 4864, 4865])
@pytest.mark.parametrize("op", ["fp64", "fp32"])
def test_sizes_against_the_batched_stepper(cuda, N, op):
    K64, K32, tab = _case(N, cuda)
    steps = 6
    one = DenseDeviceSim(K64 if op == "fp64" else K32, initial_state(tab, 1e-6, 1e-9), mu=MU, Cs=CS, V0=1e-6, Vpl=1e-9)
    ens = Ensemble(K64 if op == "fp64" else K32.double(), tab[None], mu=MU, Cs=CS, precision="fp64", max_steps=steps)
    h, t, c = one.step(steps)
    ens.iterate(3 * steps)
    r = ens.read_ctrl()[0]
    assert r.steps == steps == c.steps_done and r.attempts == c.attempts
    assert abs(r.time - c.time) <= 1e-9 * c.time and abs(t[-1] - h.sum()) <= 1e-12 * c.time
    for k in ("Tno", "Tt1o", "state", "slipv1", "slip1", "slipv"):
        a, b = one.t[k], ens.t[k][0]
        assert float(torch.linalg.norm(a - b)) <= 1e-9 * float(torch.linalg.norm(b)), k
    v = one.t["slipv"].clamp(min=1e-30)
    assert c.maxv == float(v.max())
    assert torch.allclose(one.t["slip"], torch.hypot(one.t["slip1"], one.t["slip2"]), rtol=1e-12, atol=0)
    assert torch.allclose(one.t["Tt"], torch.hypot(one.t["Tt1o"], one.t["Tt2o"]), rtol=1e-12, atol=0)
    assert torch.allclose(one.t["fric"], one.t["Tt"] / one.t["Tno"], rtol=1e-12, atol=0)
    assert torch.allclose(one.t["rake"], torch.atan2(one.t["slipv2"], one.t["slipv1"]), rtol=1e-12, atol=1e-300)
