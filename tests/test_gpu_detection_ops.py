"""ROI-Align 3D and NMS 3D kernels against their CPU oracles (``oracle/detection_oracle.py``) and the reference's own
known-answer tests for NMS (reference ``tests/test_nms.py:17-50``, same inputs, same expectations), through the
reference's import surface: ``ops3d._C.nms_3d``, ``ops3d.nms_nd``, ``ops3d.RoIAlign`` / ``roi_align_3d``."""
import numpy as np
import pytest
import torch

import ops3d
from conftest import detection_golden
from ops3d import _C
from oracle import detection_oracle as oracle

pytestmark = pytest.mark.gpu


def test_nms3d_suppresses_high_iou_duplicates():
    # one high-score box duplicated 1000x: all IoUs = 1, only the top-score box remains
    box0 = torch.tensor([0, 0, 0, 100, 100, 100], device="cuda", dtype=torch.float32)
    boxes = box0.unsqueeze(0).repeat(1000, 1)
    scores = torch.cat([torch.tensor([0.9], device="cuda"), torch.zeros(999, device="cuda")])
    keep = _C.nms_3d(boxes, scores, 0.1)
    assert keep.cpu().tolist() == [0]


def test_nms3d_keeps_non_overlapping_boxes():
    box_a = torch.tensor([0, 0, 0, 10, 10, 10], device="cuda", dtype=torch.float32)
    box_b = torch.tensor([20, 20, 20, 30, 30, 30], device="cuda", dtype=torch.float32)
    keep = _C.nms_3d(torch.stack([box_a, box_b]), torch.tensor([0.6, 0.7], device="cuda"), 0.5)
    assert set(keep.cpu().tolist()) == {0, 1} and keep.cpu().tolist() == [1, 0]  # decreasing score


@pytest.mark.parametrize("n,thr", [(1, 0.5), (63, 0.3), (64, 0.3), (65, 0.3), (300, 0.1), (1000, 0.25), (2500, 0.5)])
def test_nms3d_matches_oracle(n, thr):
    gen = torch.Generator().manual_seed(n)
    centre = torch.rand(n, 3, generator=gen) * 40
    size = torch.rand(n, 3, generator=gen) * 12 + 2
    boxes = torch.cat([centre - size / 2, centre + size / 2], 1)
    scores = torch.rand(n, generator=gen)
    keep = _C.nms_3d(boxes.cuda(), scores.cuda(), thr).cpu().tolist()
    assert keep == oracle.nms3d(boxes.numpy(), scores.numpy(), thr)
    kept2, dets = ops3d.nms_nd(torch.cat([boxes, scores[:, None]], 1).cuda(), thr)
    assert kept2.cpu().tolist() == keep and dets.shape == (n, 7)


def test_nms3d_empty_and_cpu_inputs():
    assert _C.nms_3d(torch.zeros(0, 6, device="cuda"), torch.zeros(0, device="cuda"), 0.5).numel() == 0
    with pytest.raises(RuntimeError):
        _C.nms_3d(torch.zeros(2, 6), torch.zeros(2), 0.5)


def _rois(n, N, D, H, W, seed):
    gen = torch.Generator().manual_seed(seed)
    lo = torch.rand(n, 3, generator=gen) * torch.tensor([W, H, D]) * 0.6 - 1.0     # some start outside the volume
    ext = torch.rand(n, 3, generator=gen) * torch.tensor([W, H, D]) * 0.7 + 0.3
    batch = torch.randint(0, N, (n, 1), generator=gen).float()
    return torch.cat([batch, lo, lo + ext], 1)


@pytest.mark.parametrize("order", [1, 0])
@pytest.mark.parametrize("sampling_ratio", [2, 0])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_roi_align3d_matches_oracle(dtype, sampling_ratio, order):
    N, C, D, H, W = 2, 5, 6, 7, 9
    torch.manual_seed(4)
    feats = torch.randn(N, C, D, H, W)
    rois = _rois(7, N, D, H, W, seed=5)
    out_size, scale = (2, 3, 2), 0.5 if dtype == torch.float32 else 1.0
    f = feats.to(dtype).cuda().requires_grad_(True)
    r = rois.to(dtype)  # the forward reads rois in the features' dtype, as the reference does
    out = ops3d.roi_align_3d(f, r.cuda(), out_size, scale, sampling_ratio, order)
    gout = torch.randn(out.shape)
    out.backward(gout.to(dtype).cuda())
    want = oracle.roi_align3d_forward(f.detach().float().cpu().numpy(), r.float().numpy(), out_size, scale, sampling_ratio, order)
    want_g = oracle.roi_align3d_backward(gout.to(dtype).float().numpy(), r.float().numpy(), (N, C, D, H, W), scale, sampling_ratio, order)
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    assert out.shape == (7, C) + out_size and out.dtype == dtype
    assert np.abs(out.detach().float().cpu().numpy() - want).max() <= tol * max(1.0, np.abs(want).max())
    assert np.abs(f.grad.float().cpu().numpy() - want_g).max() <= tol * max(1.0, np.abs(want_g).max())


def test_roi_align_module_and_binding_contract():
    """``ops3d.RoIAlign`` (order passed at call time; nearest uses one sample per bin) and the raw binding's
    caller-allocated tensors."""
    N, C, D, H, W = 1, 3, 5, 5, 5
    feats = torch.randn(N, C, D, H, W, device="cuda")
    rois = torch.tensor([[0, 0.0, 0.0, 0.0, 4.0, 4.0, 4.0], [0, 1.0, 2.0, 0.5, 3.5, 4.5, 2.5]], device="cuda")
    layer = ops3d.RoIAlign((2, 2, 2), 1.0, sampling_ratio=2)
    for order in (1, 0):
        got = layer(feats, rois, order=order)
        want = oracle.roi_align3d_forward(feats.cpu().numpy(), rois.cpu().numpy(), (2, 2, 2), 1.0, 1 if order == 0 else 2, order)
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-5
    out = torch.full((2, C, 2, 2, 2), 7.0, device="cuda")
    _C.roi_align_3d_forward(feats, rois, out, 2, 2, 2, 1.0, 2, 1)
    assert torch.equal(out, layer(feats, rois, order=1))
    grad_in = torch.zeros(N, C, D, H, W, device="cuda")
    _C.roi_align_3d_backward(torch.ones_like(out), rois, grad_in, 2, 2, 2, 1.0, 2, 1)
    assert abs(grad_in.sum().item() - out.numel()) <= 1e-3  # interpolation weights of in-range samples sum to one
    with pytest.raises(RuntimeError):
        _C.roi_align_3d_forward(feats, rois[:, :6].contiguous(), out, 2, 2, 2, 1.0, 2, 1)


@pytest.mark.parametrize("name,z", detection_golden("roi_align3d_"), ids=lambda v: v if isinstance(v, str) else "")
def test_roi_align3d_matches_reference_kernel_fixtures(name, z):
    size = tuple(int(v) for v in z["output_size"])
    scale, ratio, order = float(z["spatial_scale"]), int(z["sampling_ratio"]), int(z["order"])
    feats = torch.from_numpy(z["features"]).cuda().requires_grad_(True)
    out = ops3d.roi_align_3d(feats, torch.from_numpy(z["rois"]).cuda(), size, scale, ratio, order)
    out.backward(torch.from_numpy(z["grad_out"]).cuda())
    assert np.abs(out.detach().cpu().numpy() - z["out"]).max() <= 1e-5
    assert np.abs(feats.grad.cpu().numpy() - z["grad_features"]).max() <= 1e-4


@pytest.mark.parametrize("name,z", detection_golden("nms3d_"), ids=lambda v: v if isinstance(v, str) else "")
def test_nms3d_matches_reference_kernel_fixtures(name, z):
    keep = _C.nms_3d(torch.from_numpy(z["boxes"]).cuda(), torch.from_numpy(z["scores"]).cuda(), float(z["threshold"]))
    assert keep.cpu().tolist() == z["keep"].tolist()


@pytest.mark.parametrize("n", [64, 129, 4033, 4500])
def test_nms3d_order_of_ties_and_far_columns(n):
    """Scores with many ties, zeros of both signs, infinities and NaN (highest) from a strided tensor: the order of a stable
    descending sort.  4033 boxes and more have columns with words beyond those a sweep thread holds in registers."""
    gen = torch.Generator().manual_seed(n)
    centre = torch.rand(n, 3, generator=gen) * 14
    size = torch.rand(n, 3, generator=gen) * 12 + 2
    scores = torch.randint(-20, 20, (n,), generator=gen).float() / 10
    scores[:5] = torch.tensor([0.0, -0.0, float("inf"), float("-inf"), float("nan")])
    dets = torch.cat([centre - size / 2, centre + size / 2, scores[:, None]], 1).cuda()
    order = torch.sort(dets[:, 6], stable=True, descending=True)[1]
    boxes = dets[order, :6].cpu().numpy()
    keep = ops3d.nms_nd(dets, 0.3)[0].cpu()
    ranked = oracle.nms3d(boxes, -np.arange(n, dtype=np.float32), 0.3)   # already in score order
    assert keep.tolist() == order.cpu()[ranked].tolist()


@pytest.mark.parametrize("separable", ["1", "2"])                                  # by size (the smaller ones element by element), always
@pytest.mark.parametrize("size", [(1, 1, 1), (2, 5, 7), (3, 2, 31), (2, 1, 33)])   # rows of bins: one, 4 of a warp, one lane idle, too wide
@pytest.mark.parametrize("width", [8, 9, 40])                                      # 16-byte reductions or not; more than 32 vectors
def test_roi_align3d_row_shapes(size, width, separable, fda_env):
    fda_env(FDA_ROI_SEPARABLE=separable)
    N, C, D, H = 2, 9, 5, 6
    gen = torch.Generator().manual_seed(width)
    feats = torch.randn(N, C, D, H, width * (4 if width == 40 else 1), generator=gen)
    rois = torch.cat([_rois(3, N, D, H, feats.shape[4], seed=width), torch.tensor([[0, -40.0, -40, -40, -30, -30, -30], [1, 0, 0, 0, 300, 5, 4]])])
    f = feats.cuda().requires_grad_(True)
    for ratio in (2, 0):
        out = ops3d.roi_align_3d(f, rois.cuda(), size, 1.0, ratio, 1)
        gout = torch.randn(out.shape, generator=gen)
        (grad,) = torch.autograd.grad(out, f, gout.cuda())
        want = oracle.roi_align3d_forward(feats.numpy(), rois.numpy(), size, 1.0, ratio, 1)
        want_g = oracle.roi_align3d_backward(gout.numpy(), rois.numpy(), tuple(feats.shape), 1.0, ratio, 1)
        assert np.abs(out.detach().cpu().numpy() - want).max() <= 1e-4 * max(1.0, np.abs(want).max())
        assert np.abs(grad.cpu().numpy() - want_g).max() <= 1e-4 * max(1.0, np.abs(want_g).max())


@pytest.mark.parametrize("separable", ["0", "2"])
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("width", [32, 33])    # 16-byte reductions or not
@pytest.mark.parametrize("size,ratio", [((3, 3, 3), 2), ((2, 3, 1), 1), ((7, 7, 7), 2), ((2, 2, 2), 0)])   # gaps between samples, or none
def test_roi_align3d_infinities_stay_where_samples_touch(size, ratio, width, order, separable, fda_env):
    """Infinities and NaN in the features or the output gradient reach what the samples' eight corners reach and nothing else,
    the corners of weight zero among them."""
    fda_env(FDA_ROI_SEPARABLE=separable)
    N, C, D, H = 1, 5, 9, 17
    gen = torch.Generator().manual_seed(width)
    rois = torch.tensor([[0, 0.3, 0.2, 0.1, 31.4, 16.3, 8.2], [0, 3.1, 2.3, 1.4, 12.7, 9.9, 5.2], [0, 20.2, 1.1, 2.3, 23.1, 15.2, 7.7]])
    bad = torch.tensor([float("inf"), float("-inf"), float("nan")])
    feats = torch.randn(N, C, D, H, width, generator=gen)
    hit = torch.rand(feats.shape, generator=gen) < 0.01
    feats[hit] = bad[torch.randint(0, 3, (int(hit.sum()),), generator=gen)]
    f = feats.cuda().requires_grad_(True)
    out = ops3d.roi_align_3d(f, rois.cuda(), size, 1.0, ratio, order)
    gout = torch.randn(out.shape, generator=gen)
    hit = torch.rand(gout.shape, generator=gen) < 0.05
    gout[hit] = bad[torch.randint(0, 3, (int(hit.sum()),), generator=gen)]
    (grad,) = torch.autograd.grad(out, f, gout.cuda())
    with np.errstate(invalid="ignore"):
        want = oracle.roi_align3d_forward(feats.numpy(), rois.numpy(), size, 1.0, ratio, order)
        want_g = oracle.roi_align3d_backward(gout.numpy(), rois.numpy(), tuple(feats.shape), 1.0, ratio, order)
    for got, ref in ((out.detach().cpu().numpy(), want), (grad.cpu().numpy(), want_g)):
        ok = np.isfinite(ref)
        assert (np.isfinite(got) == ok).all() and ok.any() and not ok.all()
        assert np.abs(got[ok] - ref[ok]).max() <= 1e-4 * max(1.0, np.abs(ref[ok]).max())


def test_roi_align3d_small_and_large_calls_agree(fda_env):
    """Calls on both sides of the size at which the separable form takes over (16 M corners forward, 3 M backward)."""
    gen = torch.Generator().manual_seed(3)
    C, n, volume = 16, 47, (6, 12, 20)
    feats = torch.randn(1, C, *volume, generator=gen).cuda().requires_grad_(True)
    rois = _rois(n, 1, *volume, seed=9).cuda()
    for size in ((4, 4, 4), (6, 6, 6), (7, 7, 7)):   # 3.08, 10.4 and 16.5 M
        gout = torch.randn(n, C, *size, generator=gen).cuda()
        results = []
        for mode in ("1", "0", "2"):
            fda_env(FDA_ROI_SEPARABLE=mode)
            out = ops3d.roi_align_3d(feats, rois, size, 1.0, 2, 1)
            results.append((out.detach(), torch.autograd.grad(out, feats, gout)[0]))
        for out, grad in results[1:]:
            assert torch.allclose(out, results[0][0], atol=1e-5) and torch.allclose(grad, results[0][1], atol=1e-4)
