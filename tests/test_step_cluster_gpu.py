"""Attempt, decision and update of a small mesh's runs by one cluster per run
(pq3d_batch_iterate) against the separate kernels (iterate_begin and
iterate_end): the same bits of every state array and control record, for sizes
at the edges of a warp, a block, a cluster and the rule, with rejected
attempts, finished and inactive runs, directly and from a CUDA graph."""
import numpy as np
import pytest
import torch

from pyquake3d_gb300 import mesh
from pyquake3d_gb300.ensemble import Ensemble, PackedOperator
from pyquake3d_gb300.hmatrix import HMatrix

pytestmark = pytest.mark.gpu
MU, CS = 32038120320.0, 3464.0


def _tables(N, B):
    rng = np.random.default_rng(N + B)
    t = np.zeros((B, N, 10))
    t[:, :, 0] = rng.uniform(-0.3, 0.3, (B, N))
    t[:, :, 1], t[:, :, 2], t[:, :, 3], t[:, :, 4] = 0.01, 0.015, 0.1, 0.6
    t[:, :, 6] = rng.uniform(20.0, 50.0, (B, N))
    t[:, :, 7] = 10 ** rng.uniform(-10, -2, (B, N))
    return t


def _run(op, tabs, precision, how):
    e = Ensemble(op, tabs, mu=MU, Cs=CS, precision=precision, nsplit=None if precision == "hmat" else 1, dttry=1e2,
                 max_steps=5)
    if e.B > 2:
        e.deactivate(1)
    for k in range(40):
        if how == "end":
            e.begin()
            e.end()
        elif how == "iterate" or k == 0:
            e.iterate(1)
        elif k == 1:
            e.capture(39)
            e.replay()
    return e


@pytest.mark.parametrize("precision", ["bf16x6", "fp32"])
@pytest.mark.parametrize("N,B", [(1, 1), (31, 2), (33, 5), (256, 16), (257, 16), (512, 40), (700, 64), (1025, 3),
                                 (2048, 16), (2049, 2), (3001, 9), (4096, 1), (4097, 1), (2000, 17)])
def test_cluster_step_matches_the_separate_kernels(cuda, N, B, precision):
    g = torch.Generator(device=cuda).manual_seed(N)
    K = torch.randn((3 * N, 2 * N), generator=g, dtype=torch.float64, device=cuda) * 1e5
    K[torch.arange(3 * N, device=cuda), torch.arange(3 * N, device=cuda) // 3 * 2] += 1e7
    op = PackedOperator(K) if precision == "bf16x6" else K.float()
    tabs = _tables(N, B)
    a, b, c = (_run(op, tabs, precision, how) for how in ("iterate", "end", "graph"))
    assert any(r.attempts > r.steps for r in a.read_ctrl())
    assert any(r.active == 0 for r in a.read_ctrl())
    for e in (b, c):
        assert torch.equal(a.ctrl_t, e.ctrl_t)
        for k in ("Tno", "Tt1o", "Tt2o", "state", "slipv1", "slipv2", "slipv", "slip1", "slip2"):
            assert torch.equal(a.t[k], e.t[k]), k
        assert torch.equal(a.vop, e.vop)


def test_cluster_step_with_the_hierarchical_product(cuda):
    nodes, tris = mesh.rough_fault(24.0, 12.0, 30, 15, seed=2, ratio=5e-3)
    H = HMatrix(nodes, np.ascontiguousarray(tris[:850]), MU, MU, device=cuda)
    a, b = (_run(H, _tables(850, 4), "hmat", how) for how in ("iterate", "end"))
    assert torch.equal(a.ctrl_t, b.ctrl_t) and torch.equal(a.vop, b.vop)
    for k in ("Tno", "state", "slipv", "slip1"):
        assert torch.equal(a.t[k], b.t[k]), k
