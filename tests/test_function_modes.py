"""What has to see the operators' autograd Functions themselves and not the C++ graph node behind ``apply``.  No device needed: a
stand-in for the binding computes on CPU; its node entry points behave like the compiled ones (an output without history)."""
import pytest
import torch
from torch.autograd import forward_ad

import ops3d.roi_align_nd as roi_mod
import ops3d_b200.dcnv4 as dcn_mod
import ops3d_b200.flash_deform_attn as attn_mod


class Binding:
    """Per operator: output = s * ones with s the sum of the first input; counts the calls of the node entry points."""
    nodes = 0

    def _node(self, first, shape):
        self.nodes += 1
        with torch.no_grad(), torch._C._DisableTorchDispatch():
            return torch.full(shape, float(first.detach().double().sum()))

    def flash_deform_attn(self, value, shapes, lsi, packed, step, K, use_reg):
        return self._node(value, (value.shape[0], packed.shape[1], value.shape[2] * value.shape[3]))

    def flash_deform_attn_forward(self, value, shapes, lsi, packed, step, K, d_stride, threads, use_reg):
        return value.sum() * torch.ones(value.shape[0], packed.shape[1], value.shape[2] * value.shape[3])

    def flash_deform_attn_backward(self, value, shapes, lsi, packed, grad, step, K, d_stride, threads):
        return grad.sum() * torch.ones_like(value), torch.zeros_like(packed)

    def dcnv4(self, value, offset, *args):
        return self._node(value, tuple(value.shape))

    def dcnv4_forward(self, value, offset, *args):
        assert len(args) == 12 + 4 + 4
        return value.sum() * torch.ones_like(value)

    def dcnv4_backward(self, value, offset, *args):
        assert len(args) == 12 + 4 + 1 + 4
        return args[16].sum() * torch.ones_like(value), torch.zeros_like(offset)

    def roi_align_3d(self, features, rois, d, h, w, scale, ratio, order):
        return self._node(features, (rois.shape[0], features.shape[1], d, h, w))

    def roi_align_3d_forward(self, features, rois, output, d, h, w, scale, ratio, order):
        output.copy_(features.sum().expand_as(output))

    def roi_align_3d_backward(self, grad, rois, out, d, h, w, scale, ratio, order):
        out.add_(grad.sum())


@pytest.fixture
def binding(monkeypatch):
    fake = Binding()
    for mod in (attn_mod, dcn_mod, roi_mod):
        monkeypatch.setattr(mod, "_C", fake)
    return fake


def _attention():
    shapes, lsi = torch.tensor([[2, 2, 2]]), torch.tensor([0])
    packed = torch.rand(1, 3, 2, 16)
    return attn_mod.FlashDeformAttnFunction, torch.rand(1, 8, 2, 8), lambda f, v: f(v, shapes, lsi, packed, 64, 4)


def _dcnv4():
    offset, one = torch.rand(1, 2, 2, 2, 8), (1, 1, 1)
    return dcn_mod.DCNv4Function, torch.rand(1, 2, 2, 2, 8), lambda f, v: f(v, offset, one, one, (0, 0, 0), one, 1, 8, 1.0)


def _roi_align():
    rois = torch.tensor([[0, 0.0, 0, 0, 1, 1, 1]])
    return roi_mod.RoIAlign3DFunction, torch.rand(1, 2, 2, 2, 2), lambda f, v: f(v, rois, (2, 1, 1), 1.0)


OPS = [_attention, _dcnv4, _roi_align]


@pytest.mark.parametrize("make", OPS)
def test_plain_calls_take_the_node_and_subclasses_the_function(make, binding):
    function, x, call = make()
    call(function.apply, x)
    assert binding.nodes == 1

    class Mine(function):
        pass

    x.requires_grad_(True)
    out = call(Mine.apply, x)
    assert binding.nodes == 1
    (grad,) = torch.autograd.grad(out.sum(), x)
    assert torch.equal(grad, torch.full_like(x, out.numel()))


@pytest.mark.parametrize("make", OPS)
def test_forward_mode_raises(make, binding):
    function, x, call = make()
    with forward_ad.dual_level():
        dual = forward_ad.make_dual(x, torch.ones_like(x))
        with pytest.raises(NotImplementedError, match="jvp"):
            call(function.apply, dual)
        assert torch.equal(call(function.apply, x), call(function.apply, x))  # plain tensors go on as usual
    assert binding.nodes == 0


@pytest.mark.parametrize("make", OPS)
@pytest.mark.parametrize("grad", [False, True])
def test_a_traced_call_runs_on_new_inputs(make, grad, binding):
    function, x, call = make()
    with torch.set_grad_enabled(grad):
        traced = torch.jit.trace(lambda v: call(function.apply, v), (x,), check_trace=False)
        assert binding.nodes == 0
        other = x + 1
        assert torch.allclose(traced(other), call(function.apply, other))
        assert not torch.allclose(traced(other), traced(x))
