"""The BF16X6 product reads the operator that the work ahead of it on the stream
wrote: packed again, or filled by the caller's own kernel, directly before an
iteration or before the product alone, without anything in between."""
import numpy as np
import pytest
import torch

from pyquake3d_gb300 import _lib
from pyquake3d_gb300.ensemble import Ensemble, PackedOperator

pytestmark = pytest.mark.gpu
MU, CS = 32038120320.0, 3464.0


def _tables(N, B):
    rng = np.random.default_rng(N + B)
    t = np.zeros((B, N, 10))
    t[:, :, 1], t[:, :, 2], t[:, :, 3], t[:, :, 4] = 0.01, 0.015, 0.1, 0.6
    t[:, :, 6] = rng.uniform(20.0, 50.0, (B, N))
    t[:, :, 7] = 10 ** rng.uniform(-10, -2, (B, N))
    return t


@pytest.mark.parametrize("writer", ["pack", "kernel"])
@pytest.mark.parametrize("N,B", [(64, 3), (700, 16), (2000, 16)])
def test_operator_written_directly_before(cuda, writer, N, B):
    L = _lib.load()
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device=cuda).manual_seed(N)
    K = [torch.randn((3 * N, 2 * N), generator=g, dtype=torch.float64, device=cuda) * 1e5 for _ in range(3)]
    images = [PackedOperator(k).data for k in K]
    other = [torch.bitwise_not(i) for i in images]

    def write(data, k):
        if writer == "pack":
            _lib.check(L.pq3d_batch_pack_operator(K[k].data_ptr(), N, data.data_ptr(), st))
        else:
            torch.bitwise_not(other[k], out=data)

    def run(direct):
        op = PackedOperator(K[0])
        ens = Ensemble(op, _tables(N, B), mu=MU, Cs=CS, precision="bf16x6", nsplit=1)
        ens.prepare()
        products = []
        for k in (1, 2, 0, 1):
            write(op.data, k)
            if not direct:
                torch.cuda.synchronize()
            ens.iterate(1)
            write(op.data, (k + 1) % 3)
            if not direct:
                torch.cuda.synchronize()
            _lib.check(L.pq3d_batch_gemm_bf16x6(op.data.data_ptr(), ens.vop.data_ptr(), N, B, 1, 0,
                                                ens.t["rates"].data_ptr(), ens.ws.data_ptr(), ens.ws.numel(), st))
            products.append(ens.t["rates"].clone())
        torch.cuda.synchronize()
        assert ens.error_word() == 0
        return ens, products

    (a, pa), (b, pb) = run(True), run(False)
    for x, y in zip(pa, pb):
        assert torch.equal(x, y)
    assert torch.equal(a.ctrl_t, b.ctrl_t)
    for k in ("Tno", "Tt1o", "Tt2o", "state", "slipv1", "slipv2", "slipv"):
        assert torch.equal(a.t[k], b.t[k]), k
