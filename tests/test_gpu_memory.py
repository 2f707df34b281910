"""Backward calls whose fastest path needs more memory than is left take a path that fits."""
import pytest
import torch

from ops3d import _C
from ops3d_b200 import capi
from oracle import dcnv4_oracle, fda_oracle

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.fixture
def left_over():
    """``left_over(bytes)``: from here on the allocator may take that much more and then reports that memory is out."""
    total = torch.cuda.get_device_properties(0).total_memory

    def limit(size):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + size) / total)

    yield limit
    torch.cuda.set_per_process_memory_fraction(1.0)


def _attention(D):
    shapes, G, K = [(16, 32, 64), (8, 16, 32)], 8, 8
    Q = 36864
    value, sh, lsi, packed, grad_out = fda_oracle.make_inputs(shapes, 1, Q, G, D, K, seed=3)
    return value.to("cuda", torch.bfloat16), sh.cuda(), lsi.cuda(), packed.cuda(), grad_out.to("cuda", torch.bfloat16), K


def _close(got, want, ulp):
    for a, b in zip(got, want):
        a, b = a.cpu().float(), b.cpu().float()   # memory on the device may be out
        assert ((a - b).abs() <= 2 * ulp * b.abs() + 2e-5 * b.abs().max()).all()   # one rounding, sums in another order, on both sides


@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("entry", ["binding", "capi"])
def test_attention_backward_without_room_for_the_list(entry, D, left_over, fda_env):
    v, sh, lsi, pk, go, K = _attention(D)
    fda_env(FDA_BWD_SORT="0")
    want = capi.backward(v, sh, lsi, pk, go, K)
    fda_env(FDA_BWD_SORT="2")
    lists = capi.workspace_bytes(v, pk, K) - v.numel() * 4
    assert lists > 200 * MB
    left_over(v.numel() * 6 + pk.numel() * 4 + 80 * MB)   # both gradients, the image, and rounding to whole blocks
    if entry == "binding":
        got = _C.flash_deform_attn_backward(v, sh, lsi, pk, go, 64, K, 1, 0)
    else:
        got = capi.backward(v, sh, lsi, pk, go, K)
    _close(got, want, 2.0 ** -8)


def test_attention_backward_with_every_size_of_workspace(fda_env):
    """The list, the slab lists, the image alone; less than the image is refused."""
    fda_env(FDA_L2_KEEP_FRACTION="0.00001", FDA_BIN_SLAB_MB="0.02", FDA_BWD_SORT="2")
    v, sh, lsi, pk, go, K = _attention(32)
    image = v.numel() * 4
    binned = int(capi.load().fda_backward_scratch_bytes(1, v.shape[1], 8, 32, 2, pk.shape[1], K, 0))
    assert 0 < binned < capi.workspace_bytes(v, pk, K) - image
    results = []
    for size in (capi.workspace_bytes(v, pk, K), image + binned, image):
        ws = torch.full((size,), 0x7f, dtype=torch.uint8, device="cuda")
        results.append(capi.backward(v, sh, lsi, pk, go, K, workspace=ws))
    _close(results[1], results[0], 2.0 ** -8)
    _close(results[2], results[0], 2.0 ** -8)
    with pytest.raises(capi.FdaError) as info:
        capi.backward(v, sh, lsi, pk, go, K, workspace=torch.empty(image - 256, dtype=torch.uint8, device="cuda"))
    assert info.value.status == 8


@pytest.mark.parametrize("entry", ["binding", "capi"])
def test_dcnv4_backward_without_room_for_the_list(entry, left_over, fda_env):
    one, three = (1, 1, 1), (3, 3, 3)
    value, rows, grad_out = dcnv4_oracle.make_inputs(1, (24, 32, 32), 8, 16, three, one, one, one, 0, seed=2)
    value, rows, grad_out = (t.to("cuda", torch.float16).contiguous() for t in (value, rows, grad_out))
    args = (three, one, one, one, 8, 16, 1.0, 0, True)
    fda_env(FDA_BWD_SORT="0")
    want = capi.dcnv4_backward(value, rows, grad_out, *args)
    fda_env(FDA_BWD_SORT="2")
    left_over(value.numel() * 6 + rows.numel() * 2 + 80 * MB)   # the list takes 263 MB
    if entry == "binding":
        got = _C.dcnv4_backward(value, rows, *three, *one, *one, *one, 8, 16, 1.0, 64, grad_out, 0, 8, 0, True)
    else:
        got = capi.dcnv4_backward(value, rows, grad_out, *args)
    _close(got, want, 2.0 ** -11)
