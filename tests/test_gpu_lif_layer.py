"""A LIF layer's fused kernels (knp_gb300_lif_layer_*) against plain PyTorch.

Forward: weights k/256 with |k| <= 64 and 0/1 spikes make every input sum exact in FP32 in any order, so a
PyTorch FP32 loop over the steps (the same product, sum, comparison per step) gives the same bits: spikes
and checkpoints have to be equal.

Backward: against the same recurrences in FP64 on the same spikes. dI is held as hi + lo BF16, within 2^-17
of each value; the FP32 recurrence adds a few 2^-24 per step, and the products sum rows of at most 700
terms in FP32. Relative L2 error below 2^-15 allows for both."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BETA, THETA, K = 0.875, 1.0, 25.0  # beta exact in FP32


# T at and past a half of 64 and of 128 columns, past a time tile, below and off the checkpoint
# interval; batches that leave a half, or most of one, empty; widths off 8, 64, 128 and 256.
@pytest.mark.parametrize("T,B,n_in,n_out,seg", [(1, 1, 8, 1, 8), (32, 5, 64, 128, 8), (25, 50, 700, 333, 8), (7, 37, 65, 257, 3),
                                                (64, 9, 100, 130, 8), (65, 3, 200, 40, 16), (128, 3, 33, 256, 8), (129, 2, 71, 9, 5),
                                                (300, 2, 64, 300, 8), (33, 260, 16, 513, 7)])
def test_lif_layer_against_torch(T, B, n_in, n_out, seg):
    from knp_gb300 import bptt

    g = torch.Generator(device="cuda").manual_seed(T + B + n_out)
    x = (torch.rand(T, B, n_in, generator=g, device="cuda") < 0.3).float()
    w = torch.randint(-40, 65, (n_in, n_out), generator=g, device="cuda") / 256.0 * min(1.0, 40.0 / n_in)
    w = (torch.round(w * 256) / 256).requires_grad_()
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
    assert torch.equal(s.detach(), torch.stack(ss))
    dv = torch.zeros(B, n_out, device="cuda", dtype=torch.float64)
    di = torch.empty(T, B, n_out, device="cuda", dtype=torch.float64)
    for t in range(T - 1, -1, -1):
        sg = 0.5 * K / (1 + K * (us[t].double() - THETA).abs()) ** 2
        di[t] = d[t].double() * sg + dv * (1 - THETA * sg)
        dv = BETA * di[t]
    for got, ref in ((dw, x.double().flatten(0, 1).t() @ di.flatten(0, 1)), (dx, di @ w.detach().double().t())):
        assert got.shape == ref.shape
        assert float((got.double() - ref).norm()) <= 2.0 ** -15 * float(ref.norm()) + 1e-30


@pytest.mark.parametrize("seg", [0, 17])
def test_lif_layer_refuses_bad_checkpoint_intervals(seg):
    from knp_gb300 import bptt
    from knp_gb300._capi import KnpGb300Error

    x, w = torch.zeros(4, 2, 8, device="cuda"), torch.zeros(8, 8, device="cuda")
    with pytest.raises((KnpGb300Error, ZeroDivisionError)):
        bptt.LIFLayerFn.apply(x, w, BETA, THETA, seg, False, K)


# Rows whose loads are and are not 16-byte aligned, a width with padding, both halves, an unaligned source.
@pytest.mark.parametrize("R,C,width,offset", [(3, 8, 8, 0), (5, 12, 16, 0), (4, 7, 8, 0), (33, 333, 336, 0), (6, 16, 24, 1)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_operand_rows_equal_torch(R, C, width, offset, mode):
    from knp_gb300 import bptt

    g = torch.Generator(device="cuda").manual_seed(R * C)
    x = torch.randn(R * C + offset, generator=g, device="cuda")[offset:].view(R, C)
    out = bptt.operand(x, mode, False, width)
    hi = torch.nn.functional.pad(x.to(torch.bfloat16), (0, width - C))
    lo = torch.nn.functional.pad((x - x.to(torch.bfloat16).float()).to(torch.bfloat16), (0, width - C))
    assert torch.equal(out, torch.cat([hi] + ([] if mode == 0 else [hi if mode == 1 else lo]), 1))
