"""The BF16 GEMM's CTA-pair form (256 x 256 tiles): operands whose products and sums are exact in FP32
(A in {0, 1}, B = k/256 with |k| <= 128, so a sum is a multiple of 1/256 below 2^15), so the result has
to equal the FP64 product bit for bit, whatever the order of summation."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _gemm(a, b, d):
    from knp_gb300 import _capi

    err = torch.zeros(1, device="cuda", dtype=torch.int32)
    rc = _capi.lib().knp_gb300_bf16_gemm_tn(
        ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(b.data_ptr()), ctypes.c_void_p(d.data_ptr()), a.shape[0],
        b.shape[0], a.shape[1], ctypes.c_void_p(err.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, _capi.lib().knp_gb300_last_error()
    assert int(err.item()) == 0


# Whole tiles; one row and column past them; the least K; a K of exactly, and of one more than, the six
# staged chunks; several tiles per pair (both accumulators taken again); rows of D that are not 16-byte
# aligned.
@pytest.mark.parametrize("M,N,K", [(4864, 1024, 384), (4865, 1025, 8), (4864, 1025, 392), (6001, 6002, 136),
                                   (5000, 1027, 72), (39000, 512, 64)])
def test_bf16_gemm_pair_is_exact_on_dyadic_operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = (torch.rand(M, K, generator=g, device="cuda") < 0.3).to(torch.bfloat16)
    b = (torch.randint(-128, 129, (N, K), generator=g, device="cuda") / 256.0).to(torch.bfloat16)
    # Guard rows around D: nothing outside it may be written.
    buf = torch.full((M + 2, N), 7.0, device="cuda")
    _gemm(a, b, buf[1:M + 1])
    assert torch.equal(buf[1:M + 1].double(), a.double() @ b.double().t())
    assert bool((buf[0] == 7.0).all()) and bool((buf[M + 1] == 7.0).all())
