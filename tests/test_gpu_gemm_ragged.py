"""The BF16 GEMM where rows of D are no whole 16-byte units: exact on operands whose sums are exact in FP32, nothing
written outside D, and not several times slower than the next width that is."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gemm(a, b, d, err):
    from knp_gb300 import _capi

    _capi.check(_capi.lib().knp_gb300_bf16_gemm_tn(a.data_ptr(), b.data_ptr(), d.data_ptr(), a.shape[0], b.shape[0],
                                                   a.shape[1], err.data_ptr(), torch.cuda.current_stream().cuda_stream))


def _operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = (torch.rand(M, K, generator=g, device="cuda") < 0.3).to(torch.bfloat16)
    return a, (torch.randint(-128, 129, (N, K), generator=g, device="cuda") / 256.0).to(torch.bfloat16)


# Widths 1, 2 and 3 past whole units, D itself 0 to 3 elements off, a last tile of one column, of 31, of 33, of all,
# and last rows 1, 31, 33 and 129 past a tile.
@pytest.mark.parametrize("M,N", [(4865, 1025), (4895, 1055), (4897, 1057), (4993, 1279), (5000, 1026), (5121, 1031), (4864, 1028)])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_ragged_rows_are_exact_and_stay_inside(M, N, offset):
    a, b = _operands(M, N, 72)
    err = torch.zeros(1, device="cuda", dtype=torch.int32)
    buf = torch.full((M * N + 64,), 7.0, device="cuda")
    d = buf[32 + offset:32 + offset + M * N].view(M, N)
    _gemm(a, b, d, err)
    assert int(err.item()) == 0
    assert torch.equal(d.double(), a.double() @ b.double().t())
    assert bool((buf[:32 + offset] == 7.0).all()) and bool((buf[32 + offset + M * N:] == 7.0).all())


@pytest.mark.parametrize("M,N,K", [(8192, 8190, 64), (8192, 8191, 512), (1030, 8190, 128)])
def test_ragged_rows_take_about_the_time_of_whole_ones(M, N, K):
    took = []
    err = torch.zeros(1, device="cuda", dtype=torch.int32)
    for n in (N, (N + 7) // 8 * 8):
        a, b = _operands(M, n, K)
        d = torch.empty(M, n, device="cuda")
        times = []
        for _ in range(6):
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s.record()
            for _ in range(10):
                _gemm(a, b, d, err)
            e.record()
            e.synchronize()
            times.append(s.elapsed_time(e))
        took.append(min(times))
    assert took[0] < 1.9 * took[1], took
