"""Backward of a convolution layer whose saved tensors come back from a hook in another type, layout or place (GPU)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _grads(hooks, act, fp32, x_grad=True):
    from lcdrsimulator_b200.surrogate import conv
    gen = torch.Generator().manual_seed(4)
    x = torch.randn((2, 5, 6, 7, 32), generator=gen).to(torch.bfloat16).cuda().requires_grad_(x_grad)
    w = (torch.randn((16, 27, 32), generator=gen) * 0.05).cuda().requires_grad_()
    b = torch.randn((16,), generator=gen).cuda().requires_grad_()
    with torch.autograd.graph.saved_tensors_hooks(*hooks):
        y = conv.conv3d(x, w, b, act, fp32)
    gy = torch.randn(y.shape, generator=gen).to(y.dtype).cuda()
    return torch.autograd.grad(y, [x, w, b] if x_grad else [w, b], gy)


IDENTITY = (lambda t: t, lambda t: t)
OTHER_TYPE = (lambda t: t.double() if t.shape[-1] == 16 else t, lambda t: t)  # y (16 channels) comes back in FP64
STRIDED = (lambda t: t, lambda t: t.transpose(1, 2).contiguous().transpose(1, 2) if t.shape[-1] == 16 else t)
CPU = (lambda t: t.cpu(), lambda t: t.cuda())


@pytest.mark.parametrize("act, fp32", [(1, False), (1, True), (0, False)])
@pytest.mark.parametrize("hooks", [OTHER_TYPE, STRIDED, CPU], ids=["type", "strides", "cpu"])
def test_gradients_do_not_depend_on_the_hook(hooks, act, fp32):
    want = _grads(IDENTITY, act, fp32)
    got = _grads(hooks, act, fp32)
    assert torch.equal(got[0], want[0]) and torch.equal(got[2], want[2])
    # the K splits of the weight gradient are added in any order: 1e-5 of the largest entry
    assert float((got[1] - want[1]).abs().max()) <= 1e-5 * float(want[1].abs().max())


def test_weights_are_not_read_without_the_input_gradient():
    # the saved weights (16, 27, 32) come back as something that only the data gradient could object to
    hooks = (lambda t: t, lambda t: t.float() if t.dim() == 3 else t)
    want = _grads(IDENTITY, 1, False, x_grad=False)
    got = _grads(hooks, 1, False, x_grad=False)
    assert torch.equal(got[1], want[1])
    assert float((got[0] - want[0]).abs().max()) <= 1e-5 * float(want[0].abs().max())
