"""What LIFLayerFn keeps for its backward: autograd sees the tensors that the gradient is taken at, and saved-tensor
hooks get them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(x, w):
    from knp_gb300 import bptt

    return bptt.LIFLayerFn.apply(x, w, 0.9, 1.0, 8, False, 25.0)


@pytest.mark.parametrize("changed", ["weights", "spikes"])
@pytest.mark.parametrize("n_out", [64, 20])
def test_a_tensor_changed_in_place_before_the_backward_is_refused(changed, n_out):
    x = (torch.rand(6, 3, 40, device="cuda") < 0.5).float().requires_grad_()
    w = (torch.randn(40, n_out, device="cuda") * 0.3).requires_grad_()
    s = _layer(x, w)
    with torch.no_grad():
        (w if changed == "weights" else x).mul_(0.5)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        s.sum().backward()


def test_saved_tensors_pass_through_hooks():
    x = (torch.rand(6, 3, 40, device="cuda") < 0.5).float().requires_grad_()
    w = (torch.randn(40, 20, device="cuda") * 0.3).requires_grad_()
    ref = torch.autograd.grad(_layer(x, w).sum(), (x, w))
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.cuda()):
        s = _layer(x, w)
    for got, r in zip(torch.autograd.grad(s.sum(), (x, w)), ref):
        assert torch.equal(got, r)
