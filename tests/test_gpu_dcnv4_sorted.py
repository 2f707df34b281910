"""The cell-sorted backward of DCNv4-3D against the plain one, at row widths, strides and volumes around the edges of its
units, and with positions that are not finite."""
import pytest
import torch

from ops3d_b200 import capi
from oracle import dcnv4_oracle as oracle

pytestmark = pytest.mark.gpu

CASES = [  # B, (Din, Hin, Win), G, kernel, stride, pad, dilation, remove_center, scale
    (1, (1, 1, 1), 1, (1, 1, 1), (1, 1, 1), (0, 0, 0), (1, 1, 1), 0, 1.0),     # a single point
    (2, (3, 5, 4), 3, (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), 0, 1.0),     # runs of many points, border cells everywhere
    (3, (6, 7, 9), 4, (3, 3, 3), (2, 2, 2), (1, 1, 1), (1, 1, 1), 1, 0.7),
    (1, (7, 4, 11), 2, (1, 3, 5), (1, 1, 1), (0, 2, 4), (1, 2, 2), 0, 1.3),
    # a row's points crowd into few cells (not into one place: there soft-maxed mask gradients cancel to rounding noise)
    (2, (4, 9, 6), 1, (3, 3, 3), (1, 1, 1), (0, 0, 0), (1, 1, 1), 1, 0.1),
]
TYPES = [(torch.bfloat16, True), (torch.bfloat16, False), (torch.float16, True)]


def _both(fda_env, value, rows, grad_out, args):
    fda_env(FDA_BWD_SORT="0")
    plain = capi.dcnv4_backward(value, rows, grad_out, *args)
    fda_env(FDA_BWD_SORT="2")
    B, Di, Hi, Wi, _ = value.shape
    code = capi.DTYPE_CODE[value.dtype]
    kernel, stride, pad, dilation, G, D, _, rc, softmax = args
    t = capi._triple
    assert (capi.load().fda_dcnv4_backward_scratch_bytes(B, Di, Hi, Wi, G, D, t(kernel), t(stride), t(pad), t(dilation), rc, int(softmax), code)
            > capi.load().fda_dcnv4_backward_workspace_bytes(B, Di, Hi, Wi, G, D, code))
    return plain, capi.dcnv4_backward(value, rows, grad_out, *args)


@pytest.mark.parametrize("dtype,softmax", TYPES)
@pytest.mark.parametrize("D", [16, 32, 48, 64])
@pytest.mark.parametrize("case", CASES)
def test_sorted_matches_plain(case, D, dtype, softmax, fda_env):
    B, size, G, kernel, stride, pad, dilation, rc, scale = case
    value, rows, grad_out = oracle.make_inputs(B, size, G, D, kernel, stride, pad, dilation, rc, seed=D, offset_std=1.5)
    args = (kernel, stride, pad, dilation, G, D, scale, rc, softmax)
    rows = torch.nn.functional.pad(rows, (0, 3))  # padding has zero gradient
    plain, got = _both(fda_env, value.to("cuda", dtype), rows.to("cuda", dtype), grad_out.to("cuda", dtype), args)
    # either side rounds once to 16 bits and sums up to a few thousand fp32 terms in its own order
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, b in zip(plain, got):
        a, b = a.float(), b.float()
        assert ((a - b).abs() <= 2 * ulp * a.abs() + 2e-5 * a.abs().max()).all()
    assert got[1][..., -3:].abs().max().item() == 0


@pytest.mark.parametrize("dtype,softmax", TYPES)
def test_positions_that_are_not_finite(dtype, softmax, fda_env):
    B, size, G, D = 2, (4, 5, 6), 2, 32
    one = (1, 1, 1)
    value, rows, grad_out = oracle.make_inputs(B, size, G, D, (3, 3, 3), one, one, one, 0, seed=1)
    rows = rows.to("cuda", dtype)
    flat = rows.view(-1)
    for i, bad in enumerate((float("nan"), float("inf"), -float("inf"))):
        flat[1000 + 331 * i] = bad
    rows[0, 1, 1, 1, :3] = torch.tensor([float("inf"), 0.3, float("nan")])
    args = ((3, 3, 3), one, one, one, G, D, 1.0, 0, softmax)
    plain, got = _both(fda_env, value.to("cuda", dtype), rows, grad_out.to("cuda", dtype), args)
    for a, b in zip(plain, got):
        assert torch.equal(torch.isfinite(a), torch.isfinite(b))
        ok = torch.isfinite(a)
        assert ((a - b).float().abs()[ok] <= 2 * 2.0 ** -8 * a.float().abs()[ok] + 2e-5 * a.float().abs()[ok].max()).all()
