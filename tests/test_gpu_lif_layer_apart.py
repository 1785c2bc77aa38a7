"""LIF layers whose product is taken apart from the recurrence (few samples and neurons, many inputs), and layers at the
line between the two forms, against plain PyTorch.

Forward: weights k/256 with |k| <= 64 and 0/1 spikes make every input sum exact in FP32 in any order, so an FP32 loop over
the steps gives the same bits. Backward: against the same recurrence in FP64 on the same spikes. dI is held as hi + lo
BF16, within 2^-17 of each value, the FP32 recurrence adds a few 2^-24 per step, and the products sum at most 2000
terms in FP32: relative L2 error below 2^-15."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BETA, THETA, K = 0.875, 1.0, 25.0  # beta exact in FP32


# Long sums into few tiles (1 to 16 runs of K), time tiles past the checkpoint interval, intervals of 1 to 16, last
# segments of one step, widths off 8, 64 and 256, and more tiles than half the SMs.
@pytest.mark.parametrize("T,B,n_in,n_out,seg", [
    (50, 2, 5000, 300, 8), (64, 8, 2048, 10, 8), (17, 3, 3000, 65, 16), (100, 1, 4100, 7, 5), (1, 40, 2500, 513, 8),
    (33, 5, 1999, 130, 8), (9, 30, 8000, 1, 1), (2, 160, 600, 33, 16), (12, 12, 520, 64, 8), (200, 1, 784, 10, 8),
    (65, 4, 1030, 257, 3), (687, 17, 3000, 7, 8), (256, 33, 1100, 20, 16), (4, 900, 700, 333, 8)])
def test_layers_of_many_inputs_against_torch(T, B, n_in, n_out, seg):
    from knp_gb300 import bptt

    g = torch.Generator(device="cuda").manual_seed(T + B + n_out)
    x = (torch.rand(T, B, n_in, generator=g, device="cuda") < 40.0 / n_in).float()
    w = (torch.randint(-40, 65, (n_in, n_out), generator=g, device="cuda") / 256.0).requires_grad_()
    d = torch.randn(T, B, n_out, generator=g, device="cuda")
    xg = x.clone().requires_grad_()
    s = bptt.LIFLayerFn.apply(xg, w, BETA, THETA, seg, False, K)
    dx, dw = torch.autograd.grad(s, (xg, w), d)
    bptt.check_gemm_errors()

    cur = (x.double() @ w.detach().double()).float()
    v = torch.zeros(B, n_out, device="cuda")
    us, ss = [], []
    for t in range(T):
        u = BETA * v + cur[t]
        fire = (u > THETA).float()
        v = u - THETA * fire
        us.append(u)
        ss.append(fire)
    assert torch.equal(s.detach(), torch.stack(ss)) and 0 < float(s.detach().sum()) < s.numel()
    dv = torch.zeros(B, n_out, device="cuda", dtype=torch.float64)
    di = torch.empty(T, B, n_out, device="cuda", dtype=torch.float64)
    for t in range(T - 1, -1, -1):
        sg = 0.5 * K / (1 + K * (us[t].double() - THETA).abs()) ** 2
        di[t] = d[t].double() * sg + dv * (1 - THETA * sg)
        dv = BETA * di[t]
    for got, ref in ((dw, x.double().flatten(0, 1).t() @ di.flatten(0, 1)), (dx, di @ w.detach().double().t())):
        assert float((got.double() - ref).norm()) <= 2.0 ** -15 * float(ref.norm()) + 1e-30


def _graph_us(f):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        f()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        f()
    times = []
    for _ in range(6):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(10):
            graph.replay()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b) * 100)
    return min(times)


@pytest.mark.parametrize("T,B,n_out", [(50, 2, 300), (100, 4, 100)])
def test_eight_times_the_inputs_do_not_take_several_times_as_long(T, B, n_out):
    """A sum over 5000 inputs into a few tiles is spread over the device (27 us against 22 for 625 inputs; 135 when a
    pair of CTAs takes it alone)."""
    from knp_gb300 import bptt

    took = []
    for n_in in (625, 5000):
        x = (torch.rand(T, B, n_in, device="cuda") < 0.1).float()
        w = torch.randn(n_in, n_out, device="cuda") / n_in ** 0.5

        def f():
            with torch.no_grad():
                bptt.LIFLayerFn.apply(x, w, BETA, THETA, 8, False, K)
        took.append(_graph_us(f))
    assert took[1] < 2.5 * took[0], took


@pytest.mark.parametrize("offset", [0, 1, 2, 4])
def test_gradient_rows_at_any_alignment(offset):
    """The C entry point with rows of dI that start off a 16-byte boundary: the same bits, nothing outside them."""
    import ctypes

    from knp_gb300 import _capi

    T, B, n_in, N, w2 = 50, 2, 5000, 20, 24
    g = torch.Generator(device="cuda").manual_seed(1)
    s_in = (torch.rand(T * B, n_in, generator=g, device="cuda") < 0.01).to(torch.bfloat16)
    w = torch.zeros(n_in, w2, device="cuda", dtype=torch.bfloat16)
    w[:, :N] = torch.randn(n_in, N, generator=g, device="cuda") * 0.3
    S = torch.empty(T, B, N, device="cuda")
    ckpt = torch.empty(7, B, N, device="cuda")
    dS = torch.randn(T, B, N, generator=g, device="cuda")
    err = torch.zeros(1, device="cuda", dtype=torch.int32)
    lib, st, f = _capi.lib(), torch.cuda.current_stream().cuda_stream, ctypes.c_float
    _capi.check(lib.knp_gb300_lif_layer_forward(s_in.data_ptr(), w.data_ptr(), S.data_ptr(), ckpt.data_ptr(), T, B, n_in,
                                                n_in, N, w2, w2, f(0.9), f(1.0), 8, err.data_ptr(), st))
    rows = []
    for at in (0, offset):
        buf = torch.full((T * B * 2 * w2 + 16,), 7.0, device="cuda", dtype=torch.bfloat16)
        _capi.check(lib.knp_gb300_lif_layer_backward(s_in.data_ptr(), w.data_ptr(), ckpt.data_ptr(), dS.data_ptr(),
                                                     buf[8 + at:].data_ptr(), T, B, n_in, n_in, N, w2, w2, f(0.9), f(1.0), 8,
                                                     f(25.0), err.data_ptr(), st))
        rows.append(buf[8 + at:8 + at + T * B * 2 * w2].clone())
        assert (buf[:8 + at] == 7.0).all() and (buf[8 + at + T * B * 2 * w2:] == 7.0).all()
    assert torch.equal(rows[0], rows[1]) and rows[0].any() and int(err.item()) == 0
