"""Performance cases: the work users have this package do, through its public entry points.

``listed()`` holds named cases from the smallest call to the largest; ``draw(rng)`` gives further cases of the same
ranges.  ``prepare`` builds what a program has in hand before the call (seeded inputs, layers), ``run`` is one pass,
``work`` the bytes and operations a pass cannot do without, ``tolerance`` how far another correct implementation of
the same precision may be off.  A case is a dict of plain values; its ``op`` names the entry point:

  attention   ops3d.FlashDeformAttnFunction.apply, and for ``train`` the gradients of value and sampling_loc_attn
  layer       ops3d_b200.msda3d.MSDeformAttn3D, and for ``train`` the gradients of its inputs and parameters
  dcnv4       ops3d_b200.dcnv4.DCNv4Function.apply, and for ``train`` the gradients of value and offsets
  roi_align   ops3d.RoIAlign, and for ``train`` the gradient of the features
  nms         ops3d.nms_nd

Level extents are written ``"16x32x64+8x16x32"`` (depth x height x width, finest level first).
"""
from __future__ import annotations

import math

import torch

from ops3d import FlashDeformAttnFunction, RoIAlign, nms_nd
from ops3d_b200.dcnv4 import DCNv4Function
from ops3d_b200.msda3d import MSDeformAttn3D

DEVICE = "cuda"
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
SIZE = {"f32": 4, "f16": 2, "bf16": 2}

# Work bounds of drawn cases, all below what the largest listed case does.
MAX_POINT_BYTES = 2 ** 31       # sampling points x bytes of one head row
MAX_VALUE_ELEMENTS = 2 ** 27    # elements of value


# ---------------------------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # A unit-sized encoder in full precision (the smallest training call): launches and host time are what counts.
        dict(name="tiny encoder f32 train", op="attention", mode="train", levels="4x8x8+2x4x4", batch=1, queries=288,
             heads=4, channels=16, points=4, value="f32", packed="f32", where="uniform"),
        # Inference of a self-attention encoder over a 128x256x512 tile at strides 16/32.
        dict(name="small encoder bf16 infer", op="attention", mode="infer", levels="8x16x32+4x8x16", batch=2,
             queries=4608, heads=8, channels=32, points=4, value="bf16", packed="f32", where="local"),
        # Object queries of a decoder looking into the pyramid of the same tile at strides 8/16/32, training.
        dict(name="decoder bf16 train", op="attention", mode="train", levels="16x32x64+8x16x32+4x8x16", batch=4,
             queries=200, heads=8, channels=32, points=4, value="bf16", packed="f32", where="clustered"),
        # The operator's default forward: four cubic levels, 64 channels per head, 16-bit offsets.
        dict(name="cubic pyramid f16 infer", op="attention", mode="infer", levels="64x64x64+32x32x32+16x16x16+8x8x8",
             batch=1, queries=4096, heads=8, channels=64, points=8, value="f16", packed="f16", where="uniform"),
        # Full-precision training on a tile whose extents, queries and batch are odd.
        dict(name="ragged f32 train", op="attention", mode="train", levels="19x37x53+10x19x27+5x10x14", batch=3,
             queries=3001, heads=4, channels=32, points=8, value="f32", packed="f32", where="uniform"),
        # The operator's default backward: 48 channels per head (three quarters of a power of two), all 16-bit.
        dict(name="cubic encoder f16 train", op="attention", mode="train", levels="64x64x64+32x32x32", batch=1,
             queries=294912, heads=8, channels=48, points=4, value="f16", packed="f16", where="uniform"),
        # Training of an encoder over a 256x512x2048 tile at strides 16/32; every query samples around its own cell.
        dict(name="medium encoder bf16 train", op="attention", mode="train", levels="16x32x128+8x16x64", batch=1,
             queries=73728, heads=8, channels=32, points=4, value="bf16", packed="f32", where="local"),
        # The benchmark's workload: the same tile at strides 8/16/32, two of them, points spread over the whole volume.
        dict(name="large encoder bf16 train", op="attention", mode="train", levels="32x64x256+16x32x128+8x16x64", batch=2,
             queries=598016, heads=8, channels=32, points=8, value="bf16", packed="f32", where="uniform"),
        # One encoder layer (projections, packing, attention, output projection), forward and backward.
        dict(name="encoder layer bf16 train", op="layer", mode="train", levels="16x32x64+8x16x32+4x8x16", batch=1,
             queries=37376, heads=8, channels=32, points=4, value="bf16"),
        # A 3x3x3 deformable convolution over a 32x64x64 volume with 8 groups of 32 channels, soft-maxed masks.
        dict(name="dcnv4 f16 train", op="dcnv4", mode="train", batch=2, volume="32x64x64", groups=8, channels=32, kernel=3,
             stride=1, softmax=True, value="f16"),
        # Second stage of a detector: 7x7x7 crops of 256 proposals from a 128-channel feature volume.
        dict(name="roi align f32 train", op="roi_align", mode="train", batch=1, channels=128, volume="16x32x64", rois=256,
             pooled=7, ratio=2, value="f32"),
        # Proposal filtering before that stage.
        dict(name="nms 4000 boxes", op="nms", boxes=4000, threshold=0.25),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_levels(rng, count, most=1.0):
    d, h, w = _log_int(rng, 2, 32 * most), _log_int(rng, 4, 64 * most), _log_int(rng, 8, 256 * most)
    out = []
    for _ in range(count):
        out.append("%dx%dx%d" % (d, h, w))
        d, h, w = -(-d // 2), -(-h // 2), -(-w // 2)
    return "+".join(out)


def _draw_attention(rng):
    while True:
        case = dict(op="attention", mode=rng.choice(["train", "train", "infer"]), levels=_draw_levels(rng, rng.randint(1, 5)),
                    batch=rng.randint(1, 4), queries=0, heads=rng.choice([4, 8, 8, 6]), channels=rng.choice([16, 32, 32, 32, 48, 64]),
                    points=rng.choice([4, 8]), value="", packed="", where="")
        case["value"], case["packed"] = rng.choice([("f32", "f32"), ("bf16", "f32"), ("bf16", "f32"), ("bf16", "bf16"), ("f16", "f32"),
                                                    ("f16", "f16")])
        cells = sum(d * h * w for d, h, w in _levels(case))
        if rng.random() < 0.35:
            case["queries"], case["where"] = _log_int(rng, 50, 1500), rng.choice(["clustered", "uniform"])
        else:
            case["queries"], case["where"] = cells, rng.choice(["local", "uniform"])
        row_bytes = case["channels"] * SIZE[case["value"]]
        if (_points(case) * row_bytes <= MAX_POINT_BYTES
                and case["batch"] * cells * case["heads"] * case["channels"] <= MAX_VALUE_ELEMENTS):
            return case


def _draw_layer(rng):
    while True:
        case = dict(op="layer", mode=rng.choice(["train", "infer"]), levels=_draw_levels(rng, rng.randint(2, 4), 0.6),
                    batch=rng.randint(1, 2), queries=0, heads=8, channels=rng.choice([16, 32]), points=rng.choice([4, 8]),
                    value=rng.choice(["bf16", "bf16", "f32"]))
        cells = sum(d * h * w for d, h, w in _levels(case))
        case["queries"] = cells if rng.random() < 0.6 else _log_int(rng, 50, 1500)
        if _points(case) * case["channels"] * 4 <= MAX_POINT_BYTES // 2:
            return case


def _draw_dcnv4(rng):
    return dict(op="dcnv4", mode=rng.choice(["train", "infer"]), batch=rng.randint(1, 2),
                volume="%dx%dx%d" % (_log_int(rng, 5, 28), _log_int(rng, 9, 60), _log_int(rng, 9, 60)), groups=rng.choice([4, 8]),
                channels=rng.choice([16, 32]), kernel=3, stride=rng.choice([1, 1, 2]), softmax=rng.choice([True, False]),
                value=rng.choice(["f32", "f16", "bf16"]))


def _draw_roi_align(rng):
    return dict(op="roi_align", mode=rng.choice(["train", "infer"]), batch=rng.randint(1, 2), channels=_log_int(rng, 16, 192),
                volume="%dx%dx%d" % (_log_int(rng, 6, 24), _log_int(rng, 10, 48), _log_int(rng, 16, 80)), rois=_log_int(rng, 10, 300),
                pooled=rng.choice([3, 5, 7]), ratio=rng.choice([2, 2, 0]), value=rng.choice(["f32", "f32", "bf16", "f16"]))


def _draw_nms(rng):
    return dict(op="nms", boxes=_log_int(rng, 60, 9000), threshold=rng.choice([0.1, 0.25, 0.3, 0.5]))


def draw(rng):
    pick = rng.choices([_draw_attention, _draw_layer, _draw_dcnv4, _draw_roi_align, _draw_nms], [8, 1, 1, 1, 1])[0]
    return pick(rng)


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------
def _extent(text):
    return tuple(int(v) for v in text.split("x"))


def _levels(case):
    return [_extent(t) for t in case["levels"].split("+")]


def _points(case):
    return case["batch"] * case["queries"] * case["heads"] * len(_levels(case)) * case["points"]


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _level_tensors(levels):
    shapes = torch.tensor(levels, dtype=torch.long, device=DEVICE)
    sizes = shapes.prod(1)
    return shapes, torch.cat((sizes.new_zeros(1), sizes.cumsum(0)[:-1]))


def _reference_points(levels, queries, batch, gen):
    """Where the queries sit, ``[batch, queries, 3]`` = (x, y, z) in [0, 1]: the centres of all cells for a
    self-attention encoder (one query per cell), random places otherwise."""
    if queries != sum(d * h * w for d, h, w in levels):
        return torch.rand(batch, queries, 3, generator=gen, device=DEVICE)
    centres = []
    for d, h, w in levels:
        z, y, x = torch.meshgrid(*[(torch.arange(n, device=DEVICE) + 0.5) / n for n in (d, h, w)], indexing="ij")
        centres.append(torch.stack([x, y, z], -1).reshape(-1, 3))
    return torch.cat(centres).expand(batch, -1, -1)


def _prepare_attention(case, seed):
    levels, gen = _levels(case), _generator(seed)
    B, Q, G, D, K, L = case["batch"], case["queries"], case["heads"], case["channels"], case["points"], len(levels)
    shapes, lsi = _level_tensors(levels)
    N = sum(d * h * w for d, h, w in levels)
    value = torch.randn(B, N, G, D, generator=gen, device=DEVICE).to(DTYPES[case["value"]])
    if case["where"] == "uniform":    # anywhere in the volume, a few outside it
        loc = torch.rand(B, Q, G, L * K * 3, generator=gen, device=DEVICE).mul_(1.1).sub_(0.05)
    elif case["where"] == "clustered":  # around an object's centre
        loc = torch.randn(B, Q, G, L * K, 3, generator=gen, device=DEVICE).mul_(0.05)
        loc = loc.add_(torch.rand(B, Q, 1, 1, 3, generator=gen, device=DEVICE)).clamp_(-0.05, 1.05)
    else:                             # a few cells around the query's own position
        loc = torch.randn(B, Q, G, L, K, 3, generator=gen, device=DEVICE).mul_(3.0)
        loc.div_(shapes.flip(-1).float()[:, None, :]).add_(_reference_points(levels, Q, B, gen)[:, :, None, None, None, :])
    packed = torch.empty(B, Q, G, L * K * 4, device=DEVICE, dtype=DTYPES[case["packed"]])
    packed[..., : L * K * 3] = loc.view(B, Q, G, L * K * 3)
    packed[..., L * K * 3:] = torch.randn(B, Q, G, L * K, generator=gen, device=DEVICE)
    state = dict(op="attention", value=value, shapes=shapes, lsi=lsi, packed=packed, K=K)
    if case["mode"] == "train":
        state["grad_out"] = torch.randn(B, Q, G * D, generator=gen, device=DEVICE).to(value.dtype)
        value.requires_grad_(True)
        packed.requires_grad_(True)
    return state


def _prepare_layer(case, seed):
    levels, gen = _levels(case), _generator(seed)
    B, Q, G, K, L = case["batch"], case["queries"], case["heads"], case["points"], len(levels)
    C, dtype = G * case["channels"], DTYPES[case["value"]]
    shapes, lsi = _level_tensors(levels)
    N = sum(d * h * w for d, h, w in levels)
    layer = MSDeformAttn3D(C, L, G, K).to(DEVICE)
    with torch.no_grad():  # as after some training: every projection depends on its input
        for linear in (layer.sampling_offsets, layer.attention_weights, layer.value_proj, layer.output_proj):
            linear.weight.copy_(torch.randn(linear.weight.shape, generator=gen, device=DEVICE) * C ** -0.5)
    layer = layer.to(dtype)
    query = torch.randn(B, Q, C, generator=gen, device=DEVICE).to(dtype)
    src = torch.randn(B, N, C, generator=gen, device=DEVICE).to(dtype)
    ref = _reference_points(levels, Q, B, gen)[:, :, None, :].expand(B, Q, L, 3).contiguous()
    state = dict(op="layer", layer=layer, query=query, src=src, ref=ref, shapes=shapes, lsi=lsi)
    if case["mode"] == "train":
        state["grad_out"] = torch.randn(B, Q, C, generator=gen, device=DEVICE).to(dtype)
        query.requires_grad_(True)
        src.requires_grad_(True)
        state["wanted"] = [query, src] + list(layer.parameters())
    return state


def _dcnv4_out(case):
    k, s = case["kernel"], case["stride"]
    return tuple((n + 2 * (k // 2) - k) // s + 1 for n in _extent(case["volume"]))


def _prepare_dcnv4(case, seed):
    gen, dtype = _generator(seed), DTYPES[case["value"]]
    B, G, D, k, s = case["batch"], case["groups"], case["channels"], case["kernel"], case["stride"]
    padded = -(-(G * k ** 3 * 4) // 8) * 8
    out = _dcnv4_out(case)
    value = torch.randn(B, *_extent(case["volume"]), G * D, generator=gen, device=DEVICE).to(dtype)
    offset = torch.randn(B, *out, padded, generator=gen, device=DEVICE).to(dtype)
    state = dict(op="dcnv4", value=value, offset=offset,
                 args=((k,) * 3, (s,) * 3, (k // 2,) * 3, (1, 1, 1), G, D, 1.0, 64, 0, case["softmax"]))
    if case["mode"] == "train":
        state["grad_out"] = torch.randn(B, *out, G * D, generator=gen, device=DEVICE).to(dtype)
        value.requires_grad_(True)
        offset.requires_grad_(True)
    return state


def _prepare_roi_align(case, seed):
    gen, dtype = _generator(seed), DTYPES[case["value"]]
    B, C, n, p = case["batch"], case["channels"], case["rois"], case["pooled"]
    d, h, w = _extent(case["volume"])
    features = torch.randn(B, C, d, h, w, generator=gen, device=DEVICE).to(dtype)
    size = torch.tensor([w, h, d], device=DEVICE, dtype=torch.float32)
    # boxes of an eighth to a half of the volume along each axis, inside it
    extent = (0.125 + 0.375 * torch.rand(n, 3, generator=gen, device=DEVICE)) * size
    low = torch.rand(n, 3, generator=gen, device=DEVICE) * (size - extent)
    batch = torch.randint(0, B, (n, 1), generator=gen, device=DEVICE).float()
    state = dict(op="roi_align", features=features, rois=torch.cat([batch, low, low + extent], 1),
                 layer=RoIAlign((p, p, p), 1.0, sampling_ratio=case["ratio"]))
    if case["mode"] == "train":
        state["grad_out"] = torch.randn(n, C, p, p, p, generator=gen, device=DEVICE).to(dtype)
        features.requires_grad_(True)
    return state


def _prepare_nms(case, seed):
    gen, n = _generator(seed), case["boxes"]
    # about a dozen boxes compete for every place
    side = 10.0 * max(1.0, n / 12.0) ** (1.0 / 3.0)
    centre = torch.rand(n, 3, generator=gen, device=DEVICE) * side
    size = torch.rand(n, 3, generator=gen, device=DEVICE) * 12 + 2
    scores = torch.rand(n, 1, generator=gen, device=DEVICE)
    return dict(op="nms", dets=torch.cat([centre - size / 2, centre + size / 2, scores], 1), threshold=case["threshold"])


_PREPARE = dict(attention=_prepare_attention, layer=_prepare_layer, dcnv4=_prepare_dcnv4, roi_align=_prepare_roi_align,
                nms=_prepare_nms)


def prepare(case, seed):
    return _PREPARE[case["op"]](case, seed)


# ---------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------
def _forward(state):
    op = state["op"]
    if op == "attention":
        return FlashDeformAttnFunction.apply(state["value"], state["shapes"], state["lsi"], state["packed"], 64, state["K"])
    if op == "layer":
        return state["layer"](state["query"], state["ref"], state["src"], state["shapes"], state["lsi"])
    if op == "dcnv4":
        return DCNv4Function.apply(state["value"], state["offset"], *state["args"])
    return state["layer"](state["features"], state["rois"])


def _wanted(state):
    op = state["op"]
    if op == "attention":
        return [state["value"], state["packed"]]
    if op == "layer":
        return state["wanted"]
    if op == "dcnv4":
        return [state["value"], state["offset"]]
    return [state["features"]]


def run(state):
    if state["op"] == "nms":
        keep, dets = nms_nd(state["dets"], state["threshold"])
        return torch.nn.functional.pad(keep, (0, dets.shape[0] - keep.shape[0]), value=-1)   # a batch of fixed length
    if "grad_out" not in state:
        with torch.no_grad():
            return _forward(state)
    out = _forward(state)
    return [out.detach(), *torch.autograd.grad(out, _wanted(state), state["grad_out"])]


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------
def work(case):
    op, train = case["op"], case.get("mode") == "train"
    if op == "nms":
        n = case["boxes"]
        return {"bytes": n * 7 * 4 + n * 8, "flops": n * (n - 1) / 2 * 20}
    sv = SIZE[case["value"]]
    if op == "roi_align":
        d, h, w = _extent(case["volume"])
        features = case["batch"] * case["channels"] * d * h * w
        outputs = case["rois"] * case["channels"] * case["pooled"] ** 3
        samples = outputs * (case["ratio"] or 2) ** 3
        passes = 2 if train else 1   # features read / gradient written; crops written / their gradient read
        return {"bytes": passes * (features + outputs) * sv + case["rois"] * 28, "flops": passes * samples * 16}
    if op == "dcnv4":
        B, GD, K = case["batch"], case["groups"] * case["channels"], case["kernel"] ** 3
        d, h, w = _extent(case["volume"])
        cells = math.prod(_dcnv4_out(case))
        value, rows, offset = B * d * h * w * GD, B * cells * GD, B * cells * case["groups"] * K * 4
        passes = 2 if train else 1   # value, offsets, output, and the gradient of each
        points = B * cells * case["groups"] * K
        return {"bytes": passes * (value + rows + offset) * sv, "flops": points * 16 * case["channels"] * (3 if train else 1)}
    levels = _levels(case)
    B, Q, G, D, L, K = case["batch"], case["queries"], case["heads"], case["channels"], len(levels), case["points"]
    N, points, passes = sum(d * h * w for d, h, w in levels), _points(case), 2 if train else 1
    touched = min(N, 8 * Q * L * K)   # rows of value that the points can reach
    flops = points * 16 * D * (3 if train else 1)
    if op == "attention":
        # value read (and its gradient written whole); offsets and logits; output
        return {"bytes": B * G * D * (touched + (N if train else 0)) * sv + points * 4 * SIZE[case["packed"]] * passes
                + B * Q * G * D * sv * passes, "flops": flops}
    C = G * D
    weights = 2 * C * C + C * G * L * K * 4
    gemm = 2 * B * (N * C * C + Q * C * (G * L * K * 4) + Q * C * C)
    return {"bytes": passes * ((B * N * C + 2 * B * Q * C + weights) * sv) + B * Q * L * 3 * 4,
            "flops": flops + gemm * (3 if train else 1)}


def tolerance(case):
    if case["op"] == "nms":
        return "exact"
    if case["value"] != "f32":
        return {"rel": 1e-2}    # results rounded to 16 bits
    # 32-bit sums in another order.  In the layer they also decide the coordinates: of a million points one or two lie so
    # close to a cell face that the last bit moves them across it, and the gradient of a coordinate jumps there.
    return {"rel": 1e-3} if case["op"] == "layer" else {"rel": 1e-5}
