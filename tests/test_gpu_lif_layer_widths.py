"""The LIF layer's C entry points with gradient rows that are wider than the layer needs: knp_gb300_lif_layer_backward
fills each half of dI up to its width, zeros from column N on."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


# The width ends in the tile of 256 columns that holds the last neuron, one past it, and several past it.
@pytest.mark.parametrize("N,w2", [(10, 64), (10, 256), (10, 264), (10, 512), (250, 1024), (300, 576)])
def test_gradient_halves_are_zero_past_the_last_neuron(N, w2):
    from knp_gb300 import _capi

    T, B, K = 9, 6, 40
    g = torch.Generator(device="cuda").manual_seed(N + w2)
    s_in = (torch.rand(T * B, K, generator=g, device="cuda") < 0.4).to(torch.bfloat16)
    w = torch.zeros(K, w2, device="cuda", dtype=torch.bfloat16)
    w[:, :N] = torch.randn(K, N, generator=g, device="cuda") * 0.3
    S = torch.empty(T, B, N, device="cuda")
    ckpt = torch.empty(2, B, N, device="cuda")
    dS = torch.randn(T, B, N, generator=g, device="cuda")
    dI = torch.full((T * B, 2 * w2), float("nan"), device="cuda", dtype=torch.bfloat16)
    ds = torch.empty(T * B, K, device="cuda")
    err = torch.zeros(1, device="cuda", dtype=torch.int32)
    lib, st = _capi.lib(), torch.cuda.current_stream().cuda_stream
    f = ctypes.c_float
    _capi.check(lib.knp_gb300_lif_layer_forward(s_in.data_ptr(), w.data_ptr(), S.data_ptr(), ckpt.data_ptr(), T, B, K, K, N,
                                                w2, w2, f(0.9), f(1.0), 8, err.data_ptr(), st))
    _capi.check(lib.knp_gb300_lif_layer_backward(s_in.data_ptr(), w.data_ptr(), ckpt.data_ptr(), dS.data_ptr(),
                                                 dI.data_ptr(), T, B, K, K, N, w2, w2, f(0.9), f(1.0), 8, f(25.0),
                                                 err.data_ptr(), st))
    hi, lo = dI[:, :w2], dI[:, w2:]
    assert not hi[:, N:].any() and not lo[:, N:].any()
    assert hi[:, :N].any() and torch.isfinite(dI.float()).all()
    if w2 % 64 == 0:
        _capi.check(lib.knp_gb300_lif_layer_ds(dI.data_ptr(), w.data_ptr(), ds.data_ptr(), T * B, K, w2, err.data_ptr(), st))
        ref = (hi.double() + lo.double()) @ w.double().t()
        # FP32 sums of 2 w2 products: at most 2 w2 roundings of 2^-24 of the terms' absolute sum.
        bound = (hi.double().abs() + lo.double().abs()) @ w.double().abs().t() * (2 * w2 * 2.0 ** -24)
        assert ((ds.double() - ref).abs() <= bound).all()
    assert int(err.item()) == 0
