"""pq3d_hmat_aca from several host threads, each on a stream of its own and gone
afterwards, and captured in a CUDA graph: the factors, ranks and states of the
call on the current stream, bit for bit, with blocks of all three kinds."""
import threading

import numpy as np
import pytest
import torch

from pyquake3d_gb300 import _lib, mesh
from pyquake3d_gb300.hmatrix import HMatrix

pytestmark = pytest.mark.gpu
MU = 32038120320.0


def test_threads_and_capture(cuda):
    L = _lib.load()
    nodes, tris = mesh.rough_fault(60.0, 6.0, 100, 10, seed=2, ratio=5e-3)
    H = HMatrix(nodes, tris, MU, MU, min_size=16, mini_leaf=16, device=cuda)
    kcap = H.kcap.cpu().numpy()
    ids = np.nonzero(kcap)[0]
    blk = H.blk.cpu().numpy()[ids]
    m, n = blk[:, 1] - blk[:, 0], blk[:, 3] - blk[:, 2]
    assert (m + n).min() < 64 and (m + n).max() > 512   # a quarter CTA's blocks and a cluster's
    need, rows = kcap[ids].astype(np.int64) * (3 * m + 2 * n), 3 * m
    dev = [torch.as_tensor(np.ascontiguousarray(a), device=cuda) for a in
           (blk, kcap[ids], np.concatenate([[0], np.cumsum(need)[:-1]]), np.concatenate([[0], np.cumsum(rows)[:-1]]))]

    def buffers():
        return (torch.zeros(int(need.sum()), dtype=torch.float64, device=cuda),
                torch.zeros(int(rows.sum()), dtype=torch.uint8, device=cuda),
                *(torch.full((len(ids),), -9, dtype=torch.int32, device=cuda) for _ in range(2)))

    def aca(b):
        return L.pq3d_hmat_aca(H.tables.data_ptr(), H.N, H.perm.data_ptr(), len(ids), dev[0].data_ptr(),
                               dev[1].data_ptr(), 1e-4, MU, MU, 0, b[0].data_ptr(), dev[2].data_ptr(), b[1].data_ptr(),
                               dev[3].data_ptr(), b[2].data_ptr(), b[3].data_ptr(),
                               torch.cuda.current_stream().cuda_stream)

    ref = buffers()
    _lib.check(aca(ref))
    torch.cuda.synchronize()
    assert (ref[2] > 0).all() and (ref[3] == 0).all()
    got, rcs = [buffers() for _ in range(6)], []
    torch.cuda.synchronize()

    def work(b):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            rcs.append(aca(b))
        s.synchronize()

    threads = [threading.Thread(target=work, args=(b,)) for b in got]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert rcs == [_lib.PQ3D_OK] * 6
    b = buffers()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        assert aca(b) == _lib.PQ3D_OK
    for _ in range(2):
        for t, v in zip(b, (0, 0, -9, -9)):
            t.fill_(v)
        g.replay()
        torch.cuda.synchronize()
        got.append(tuple(t.clone() for t in b))
    for b in got:
        for x, y in zip(ref, b):
            assert torch.equal(x, y)
