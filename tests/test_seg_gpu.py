"""The tiled full-space assembly (edge matrices shared by the triangles of a
tile, csrc/seg_device.cuh) against the oracle's operator, whose pairs are the
published angular dislocations: sizes at the edges of a tile, meshes whose
triangles share nothing, receivers on an edge of a source, sources of zero
area, and a Lame pair with nu != 1/4.  Tolerance: the project's parity bar,
1e-10 of a receiver row's largest entry (FP64 rounding of either formula is
below 1e-12 of it on these meshes)."""
import numpy as np
import pytest
import torch

import oracle
from pyquake3d_gb300 import gf, mesh
from pyquake3d_gb300.gf import join_ops

pytestmark = pytest.mark.gpu
MU = 32038120320.0


def _check(nodes, tris, lam, cuda, rows=None):
    K64, K32 = gf.assemble_dense(nodes, tris, MU, lam, device=cuda, rows=rows)
    ref = join_ops(dict(zip(oracle.OPS, oracle.assemble_dense(nodes, tris, MU, lam))))
    if rows is not None:
        ref = ref[3 * rows[0]:3 * rows[1]]
    got = K64.cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    # one scale per receiver: its three traction rows together
    g, r = (np.nan_to_num(m).reshape(len(ref) // 3, -1) for m in (got, ref))
    assert np.all(np.abs(g - r).max(1) <= 1e-10 * np.abs(r).max(1))
    assert torch.equal(K32.nan_to_num(), K64.float().nan_to_num())


@pytest.mark.parametrize("N", [1, 2, 31, 255, 256, 257, 513])
@pytest.mark.parametrize("order", ["mesh", "shuffled", "soup"])
def test_tile_edges(cuda, N, order):
    nodes, tris = mesh.rough_fault(18.0, 15.0, 18, 15, seed=3, ratio=5e-3)
    rng = np.random.default_rng(N)
    if order == "shuffled":
        tris = tris[rng.permutation(len(tris))]
        tris = np.take_along_axis(tris, (np.arange(3)[None] + rng.integers(0, 3, (len(tris), 1))) % 3, 1)
    if order == "soup":   # no vertex in common: 3 N vertices and edges
        nodes, tris = nodes[tris.ravel() - 1], np.arange(1, 3 * len(tris) + 1).reshape(-1, 3)
    _check(nodes, np.ascontiguousarray(tris[:N]), MU, cuda)


@pytest.mark.parametrize("rows", [(0, 1), (7, 40), (299, 300)])
def test_row_range_and_other_poisson_ratio(cuda, rows):
    nodes, tris = mesh.rough_fault(15.0, 10.0, 15, 10, seed=4, ratio=5e-3)
    _check(nodes, tris, 0.6 * MU, cuda, rows)


def test_receivers_on_edges_and_sources_without_area(cuda):
    """The centroid of element 2 lies on an edge of element 1 in its plane
    (the configuration test gives zero strain), that of element 3 on the same
    line beyond the edge, element 4 has no area (NaN), element 5 is flat
    (strike axis e_Y)."""
    nodes = 1e3 * np.array([[0, 0, 0], [3, 0, 0], [0, 0, 3], [1, 0, -1], [2, 0, -1], [1.5, 0, 2], [4, 0, -1],
                            [5, 0, -1], [4.5, 0, 2], [8, 1, 0], [9, 1, 0], [10, 1, 0], [1, 4, 1], [2, 4, 1], [1, 5, 1]],
                           dtype=np.float64)
    tris = np.arange(1, 16).reshape(5, 3)
    _check(nodes, tris, MU, cuda)
    assert np.all(gf.assemble_dense(nodes, tris, MU, MU, device=cuda)[0][3:6, 0:2].cpu().numpy() == 0.0)
