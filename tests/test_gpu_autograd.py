"""The operators' graph nodes: which inputs get gradients, what is saved, and what raises."""
import pytest
import torch

from ops3d import FlashDeformAttnFunction, roi_align_3d
from ops3d_b200.dcnv4 import DCNv4Function

pytestmark = pytest.mark.gpu


def _attention():
    shapes = torch.tensor([[3, 4, 5], [2, 2, 3]], device="cuda")
    lsi = torch.tensor([0, 60], device="cuda")
    value = torch.randn(2, 72, 2, 16, device="cuda")
    packed = torch.rand(2, 7, 2, 2 * 4 * 4, device="cuda")
    return [value, packed], lambda v, p: FlashDeformAttnFunction.apply(v, shapes, lsi, p, 64, 4)


def _dcnv4():
    value, offset = torch.randn(1, 3, 4, 5, 32, device="cuda"), torch.randn(1, 3, 4, 5, 2 * 27 * 4, device="cuda")
    return [value, offset], lambda v, o: DCNv4Function.apply(v, o, (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), 2, 16, 1.0)


def _roi_align():
    rois = torch.tensor([[0, 0.0, 0, 0, 3, 3, 3], [1, 1.0, 1, 0, 4, 3, 2]], device="cuda")
    return [torch.randn(2, 3, 4, 4, 5, device="cuda")], lambda f: roi_align_3d(f, rois, (2, 2, 2), 1.0, 2, 1)


@pytest.mark.parametrize("make", [_attention, _dcnv4, _roi_align])
def test_graph_node_semantics(make):
    inputs, op = make()
    plain = op(*inputs)
    assert not plain.requires_grad
    with torch.no_grad():
        assert not op(*[t.detach().requires_grad_(True) for t in inputs]).requires_grad
    gout = torch.randn_like(plain)
    leaves = [t.clone().requires_grad_(True) for t in inputs]
    out = op(*leaves)
    assert torch.equal(out, plain) and out.requires_grad
    want = torch.autograd.grad(out, leaves, gout, retain_graph=True)
    for k, leaf in enumerate(leaves):  # one gradient at a time, from a graph that was kept
        got, = torch.autograd.grad(out, leaf, gout, retain_graph=True)
        assert torch.allclose(got, want[k], atol=1e-4 * want[k].abs().max().item())   # the order of fp32 sums
        only = [t.clone().requires_grad_(i == k) for i, t in enumerate(inputs)]
        op(*only).backward(gout)
        assert torch.allclose(only[k].grad, want[k], atol=1e-4 * want[k].abs().max().item())
        assert all(t.grad is None for i, t in enumerate(only) if i != k)
    torch.autograd.grad(out, leaves, gout)
    with pytest.raises(RuntimeError, match="backward through the graph a second time"):
        torch.autograd.grad(out, leaves, gout)
    out = op(*leaves)
    first = torch.autograd.grad(out, leaves, gout.clone().requires_grad_(True), create_graph=True)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(first[0].sum(), leaves[0])


@pytest.mark.parametrize("make", [_attention, _dcnv4])
def test_saved_inputs_are_version_checked(make):
    inputs, op = make()
    leaves = [t.clone().requires_grad_(True) for t in inputs]
    copies = [t * 1 for t in leaves]
    out = op(*copies)
    with torch.no_grad():
        copies[0].mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.sum().backward()


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, grad):
        return None


@pytest.mark.parametrize("make", [_attention, _dcnv4, _roi_align])
def test_an_output_without_a_gradient_counts_as_zeros(make):
    inputs, op = make()
    leaves = [t.clone().requires_grad_(True) for t in inputs]
    for got, leaf in zip(torch.autograd.grad(_NoGradient.apply(op(*leaves)).sum(), leaves), leaves):
        assert got.shape == leaf.shape and not got.any()


def test_an_error_message_with_numbers_raises():
    value, offset = torch.randn(1, 2, 2, 2, 32, device="cuda"), torch.randn(1, 2, 2, 2, 8, device="cuda")
    one = (1, 1, 1)
    with pytest.raises(RuntimeError, match=r"dont match: \(32 vs 24\)"):
        DCNv4Function.apply(value, offset, one, one, (0, 0, 0), one, 3, 8, 1.0)


@pytest.mark.parametrize("make", [_attention, _dcnv4, _roi_align])
def test_side_streams_and_threads(make):
    """A node's backward runs on the stream of its forward, whichever thread asks for it."""
    import threading

    inputs, op = make()
    plain = [t.clone().requires_grad_(True) for t in inputs]
    out = op(*plain)
    gout = torch.randn_like(out)
    want = torch.autograd.grad(out, plain, gout)
    torch.cuda.synchronize()
    results = [None] * 4

    def work(i):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(2_000_000)   # what the side stream does is late
            leaves = [(t * 1).requires_grad_(True) for t in inputs]
            mine = op(*leaves)
            grads = torch.autograd.grad(mine, leaves, gout * 1)
            results[i] = [mine.detach().clone()] + [g.clone() for g in grads]
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(results))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for got in results:
        assert torch.equal(got[0], out.detach())
        for a, b in zip(got[1:], want):
            assert torch.allclose(a, b, atol=1e-4 * b.abs().max().item())   # the order of fp32 sums
