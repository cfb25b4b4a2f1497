"""The tiled half-space assembly (an edge's free-surface correction shared by
its two triangles) and the point calls (pairs shared by the warps of a block,
transfers through mapped memory) against the oracle, whose pairs are the
published formulas: sizes at the edges of a tile, a block, a warp and the
mapped buffer.  Tolerance: the project's parity bar, normwise 1e-10, on
geometries without a near-vertical side (where the published formulas
themselves lose digits)."""
import numpy as np
import pytest
import torch

import oracle
from pyquake3d_gb300 import _lib, gf
from pyquake3d_gb300.gf import join_ops
from util import normwise_rel

pytestmark = pytest.mark.gpu
MU = 32038120320.0


def _fault(nx, ny, dip=60.0, h=400.0, top=0.0):
    """Plane fault of 2 nx ny triangles from the depth `top` down, its nodes
    moved a little within the plane; two triangles in the surface beside it."""
    rng = np.random.default_rng(nx)
    u, v = (a.ravel().astype(np.float64) for a in np.meshgrid(np.arange(nx + 1), np.arange(ny + 1), indexing="ij"))
    u, v = h * (u + 0.1 * rng.uniform(-1, 1, u.size)), h * (v + np.where(v > 0, 0.1 * rng.uniform(-1, 1, v.size), 0.0))
    c, s = np.cos(np.radians(dip)), np.sin(np.radians(dip))
    nodes = np.stack([u, v * c, -top - v * s], 1)
    i, j = (a.ravel() for a in np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij"))
    n = 1 + i * (ny + 1) + j
    tris = np.stack([np.stack([n, n + ny + 1, n + ny + 2], 1), np.stack([n, n + ny + 2, n + 1], 1)], 1).reshape(-1, 3)
    flat = h * np.array([[0.0, -9, 0], [2, -9, 0], [2, -7, 0], [0, -7, 0]])
    m = len(nodes)
    return np.concatenate([nodes, flat]), np.concatenate([tris, [[m + 1, m + 2, m + 3], [m + 1, m + 3, m + 4]]])


def _check(nodes, tris, lam, cuda, rows=None):
    K64, K32 = gf.assemble_dense(nodes, tris, MU, lam, halfspace=True, device=cuda, rows=rows)
    ref = join_ops(dict(zip(oracle.OPS, oracle.assemble_dense(nodes, tris, MU, lam, halfspace=True, nthreads=8))))
    if rows is not None:
        ref = ref[3 * rows[0]:3 * rows[1]]
    got = K64.cpu().numpy()
    # receivers in the surface: with nu = 1/4 no traction at all there, so the scale is that of a source's own, mu / h
    free = np.repeat((nodes[tris - 1, 2] == 0.0).all(1)[slice(*rows or (0, None))], 3)
    assert np.abs(got - ref)[free].max(initial=0.0) < 1e-10 * MU / 400.0
    assert normwise_rel(ref[~free], got[~free]) < 1e-10
    assert torch.equal(K32, K64.float())


@pytest.mark.parametrize("N", [1, 2, 239, 240, 241, 481])
@pytest.mark.parametrize("order", ["mesh", "shuffled", "soup"])
def test_tile_edges(cuda, N, order):
    nodes, tris = _fault(16, 15)
    tris = np.concatenate([tris[-2:], tris[:-2]])   # the surface triangles first
    rng = np.random.default_rng(N)
    if order == "shuffled":
        tris = tris[rng.permutation(len(tris))]
        tris = np.take_along_axis(tris, (np.arange(3)[None] + rng.integers(0, 3, (len(tris), 1))) % 3, 1)
    if order == "soup":   # no vertex in common: 3 N vertices and edges
        nodes, tris = nodes[tris.ravel() - 1], np.arange(1, 3 * len(tris) + 1).reshape(-1, 3)
    _check(nodes, np.ascontiguousarray(tris[:N]), MU, cuda)


@pytest.mark.parametrize("rows", [(0, 1), (5, 38), (241, 242)])
def test_row_range_and_other_poisson_ratio(cuda, rows):
    nodes, tris = _fault(12, 10, top=900.0)
    _check(nodes, tris, 0.6 * MU, cuda, rows)


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 4095, 4097, 4369, 4370])
def test_points_of_one_source(cuda, n, half):
    rng = np.random.default_rng(n)
    P = np.array([[0.0, 0, -1000], [1000, 100, -1100], [600, 900, -1800]])
    R = rng.uniform([-4000, -4000, -6000], [4000, 4000, 0], (n, 3))
    X, Y, Z = (np.ascontiguousarray(R[:, k]) for k in range(3))
    got = gf.TDstressFS(X, Y, Z, P[0], P[1], P[2], 1.0, -0.5, 0.3, MU, 0.8 * MU, half)
    ref = oracle.tdstress(X, Y, Z, P[0], P[1], P[2], 1.0, -0.5, 0.3, MU, 0.8 * MU, half)
    for g, r in zip(got, ref):   # (6, n) and (n, 6)
        assert normwise_rel(r, g.T) < 1e-10


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("n", [1, 33, 2730, 2731, 4096, 4097])
def test_sources_at_one_point(cuda, n, half):
    rng = np.random.default_rng(n)
    a, c = rng.uniform(0, 2 * np.pi, n), rng.uniform([-9000, -9000, -9000], [9000, 9000, -2000], (n, 3))
    P = [np.ascontiguousarray(c + np.stack([x * np.cos(a) - y * np.sin(a), x * np.sin(a) + y * np.cos(a),
                                            np.full(n, z)], 1))
         for x, y, z in ((0.0, 0.0, 0.0), (700.0, 60.0, -80.0), (400.0, 500.0, -700.0))]
    s, e = np.zeros((n, 6)), np.zeros((n, 6))
    D = _lib.c_double_p
    p = lambda v: v.ctypes.data_as(D)
    slips = 1.0, -0.5, 0.3
    _lib.load().TDstressEachSourceAtReceiver_C(100.0, -200.0, -500.0, *(p(v) for v in P), n, *slips, MU, 0.8 * MU,
                                               half, p(s), p(e))
    rs, re = oracle.tdstress_each_source(100.0, -200.0, -500.0, *P, *slips, MU, 0.8 * MU, half)
    assert normwise_rel(rs, s) < 1e-10
    assert normwise_rel(re, e) < 1e-10
