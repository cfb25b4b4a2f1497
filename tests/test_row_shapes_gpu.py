"""The dense product at the sizes where its launch changes (warps per receiver,
resident blocks of the FP32 operator) against torch in FP64: each row's error
within the rounding of its own sum of 2N products, and all of the output written."""
import pytest
import torch

from pyquake3d_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 7, 31, 32, 33, 127, 128, 304, 305, 608, 609, 1216, 1217, 1300, 2431, 2432, 2433, 3648,
                               3649, 4864, 4865, 6001])
@pytest.mark.parametrize("op", ["fp64", "fp32"])
def test_product_against_torch(cuda, N, op):
    n = 2 * N / 32 + 10   # additions one after the other: a lane's products, 5 levels of lanes, 4 parts, the reference
    L = _lib.load()
    g = torch.Generator(device=cuda).manual_seed(N)
    K = torch.randn((3 * N, 2 * N), generator=g, dtype=torch.float64, device=cuda)
    v = torch.randn(2 * N, generator=g, dtype=torch.float64, device=cuda)
    out = torch.full((3 * N,), float("nan"), dtype=torch.float64, device=cuda)
    st = torch.cuda.current_stream().cuda_stream
    if op == "fp64":
        _lib.check(L.pq3d_dense_matvec_f64(K.data_ptr(), N, v.data_ptr(), out.data_ptr(), st))
        bar = (n + 1) * 2.0 ** -53
    else:   # v per source as (hi1, hi2, lo1, lo2); the sum and its rounding errors apart, in FP32
        K = K.float()
        hi = v.float()
        lo = (v - hi.double()).float()
        vs = torch.cat([hi.view(N, 2), lo.view(N, 2)], 1).contiguous()
        _lib.check(L.pq3d_dense_matvec_f32(K.data_ptr(), N, vs.data_ptr(), out.data_ptr(), st))
        bar = n * n * 2.0 ** -48 + 2.0 ** -46
    ref = K.double() @ v
    scale = K.double().abs() @ v.abs()
    assert bool(((out - ref).abs() <= bar * scale).all())
