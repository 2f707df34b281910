"""The walk of the cell-sorted backward at every row width it takes, with runs of equal cells around the sizes of its units
(8 points) and pairs of units (16), against the CPU oracle."""
import pytest
import torch

from ops3d_b200 import capi
from oracle import fda_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vdt,pdt", [(torch.bfloat16, torch.float32), (torch.float16, torch.float16)])
@pytest.mark.parametrize("D", [16, 32, 48, 64])
@pytest.mark.parametrize("shapes,Q", [([(1, 1, 1)], 1),                # one cell: a single run of four points at most
                                      ([(2, 2, 2), (1, 2, 1)], 17),    # a few long runs, border cells on every side
                                      ([(5, 6, 7)], 150),              # runs of a few points
                                      ([(3, 5, 4), (2, 3, 2), (1, 2, 1)], 700)])
def test_walk_matches_oracle(shapes, Q, D, vdt, pdt, fda_env):
    B, G, K = 2, 3, 4
    value, sh, lsi, packed, grad_out = fda_oracle.make_inputs(shapes, B, Q, G, D, K, seed=D + Q, lo=-0.3, hi=1.3)
    v, pk, go = value.to("cuda", vdt), packed.to("cuda", pdt), grad_out.to("cuda", vdt)
    fda_env(FDA_BWD_SORT="2", FDA_SORT_GRID_X="2")
    assert capi.backward_path(v, pk, K) == (2 if D == 32 else 3)
    gv, gp = capi.backward(v, sh.cuda(), lsi.cuda(), pk, go, K)
    _, ref_gv, ref_gp = fda_oracle.fused_forward_backward(v.float().cpu(), sh, pk.float().cpu(), go.float().cpu(), K)
    # one rounding to the output type (half a unit in the last place of bf16 / fp16), and fp32 sums of up to a few thousand terms
    ulp = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 0.0}
    for got, ref, dt in ((gv, ref_gv, vdt), (gp, ref_gp, pdt)):
        bound = ulp[dt] * ref.abs() + 2e-5 * ref.abs().max()
        assert ((got.float().cpu() - ref).abs() <= bound).all()


@pytest.mark.parametrize("vdt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [16, 32, 48, 64])
@pytest.mark.parametrize("masked", [False, True])
def test_small_weights_keep_their_bits(D, vdt, masked, fda_env):
    """Cells reached only through soft-max probabilities down to 1e-14, alone or beside points of a probability near one
    whose output gradient is zero: the fp32 image must agree with the plain kernel's, relative to every element.  Output
    gradients are not negative, so nothing cancels; a cell sums at most a few hundred terms, in fp32 and in another order
    (relative error below 100 * 2^-24 in either kernel: errors of a sum of positive terms grow far slower than its length)."""
    shapes, Q, G, K = [(4, 8, 8)], 96, 2, 8
    gen = torch.Generator().manual_seed(D)
    N = 256
    sh, lsi = torch.tensor(shapes).cuda(), torch.zeros(1, dtype=torch.long).cuda()
    # voxel positions on a grid of 1/64: exact in fp32; the last point of a row, the strong one, sits left of x = 2 or anywhere
    voxel = torch.randint(0, 64 * 3, (1, Q, G, K, 3), generator=gen) / 64.0
    voxel[..., 0] += 3.5
    voxel[..., -1, 0] = torch.randint(0, 64 * (7 if masked else 2), (1, Q, G), generator=gen) / 64.0
    loc = (voxel + 0.5) / torch.tensor([8.0, 8.0, 4.0])
    logits = -20.0 - torch.rand(1, Q, G, K, generator=gen) * 12.0
    logits[..., -1] = 0.0
    packed = torch.cat([loc.reshape(1, Q, G, 3 * K), logits], -1).cuda()
    grad_out = torch.rand(1, Q, G, D, generator=gen) + 0.5
    if masked:  # rows with a gradient have small weights only
        packed[:, ::2, :, 4 * K - 1] = -33.0
        packed[:, ::2, :, 3 * K] = 0.0      # the first point is the strong one now, out of the way
        packed[:, ::2, :, 0:3] = torch.tensor([0.06, 0.06, 0.12]).cuda()
        grad_out[:, 1::2] = 0.0
    v = torch.randn(1, N, G, D, generator=gen).to("cuda", vdt)
    go = grad_out.reshape(1, Q, G * D).to("cuda", vdt)
    images = []
    for mode in ("0", "2"):
        fda_env(FDA_BWD_SORT=mode, FDA_BINNING="0")
        assert (capi.backward_path(v, packed, K) >= 2) == (mode == "2")
        scratch = torch.empty(max(256, capi.scratch_bytes(v, packed, K)), dtype=torch.uint8, device="cuda")
        image, gp = torch.empty(v.shape, dtype=torch.float32, device="cuda"), torch.empty_like(packed)
        capi.backward_accumulate_levels(v, sh, lsi, packed, go, K, image, gp, 0, 1, capi.BWD_ZERO_IMAGE | capi.BWD_FINALIZE, scratch=scratch)
        images.append(image.double())
    plain, got = images
    reached = plain > 0
    assert torch.equal(reached, got > 0) and plain[reached].min() < 1e-8
    assert ((got - plain).abs() <= 200 * 2.0 ** -24 * plain).all()


@pytest.mark.parametrize("vdt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [16, 32, 48, 64])
def test_no_further_from_64_bits_than_the_plain_kernel(D, vdt, fda_env):
    """The walk's matrix products against the plain kernel's fp32 FMAs: relative error of the fp32 image and of the packed
    gradients (positions on a grid of 1/64, exact in fp32).  Averages over 3e5 numbers and more: 5 % is far outside their spread."""
    shapes, Q, G, K = [(8, 16, 8), (4, 8, 8)], 500, 4, 8
    gen = torch.Generator().manual_seed(D)
    extent = torch.tensor([[w, h, d] for d, h, w in shapes], dtype=torch.float32)
    voxel = torch.randint(-16, 64 * 16, (1, Q, G, 2, K, 3), generator=gen) / 64.0
    loc = (voxel.remainder(extent[:, None]) + 0.5) / extent[:, None]
    logits = torch.randn(1, Q, G, 2, K, generator=gen)
    packed = torch.cat([loc.flatten(3), logits.flatten(3)], -1)
    N = sum(d * h * w for d, h, w in shapes)
    v, go = torch.randn(1, N, G, D, generator=gen).to(vdt), torch.randn(1, Q, G * D, generator=gen).to(vdt)
    v64, loc64, logits64 = (t.double().requires_grad_(True) for t in (v, loc, logits))
    out = fda_oracle.ms_deform_attn_core_pytorch_3d(v64, shapes, loc64, logits64.flatten(3).softmax(-1).view_as(logits64))
    want = torch.autograd.grad(out, (v64, loc64, logits64), go.double())
    want = [want[0], want[1].flatten(3), want[2].flatten(3)]
    sh, lsi = torch.tensor(shapes).cuda(), torch.tensor([0, 1024]).cuda()
    errors = []
    for mode in ("0", "2"):
        fda_env(FDA_BWD_SORT=mode, FDA_BINNING="0")
        args = v.cuda(), sh, lsi, packed.cuda(), go.cuda(), K
        scratch = torch.empty(max(256, capi.scratch_bytes(args[0], args[3], K)), dtype=torch.uint8, device="cuda")
        image, gp = torch.empty(v.shape, dtype=torch.float32, device="cuda"), torch.empty(packed.shape, device="cuda")
        capi.backward_accumulate_levels(*args, image, gp, 0, 2, capi.BWD_ZERO_IMAGE | capi.BWD_FINALIZE, scratch=scratch)
        got = [image, gp[..., :48], gp[..., 48:]]
        errors.append([((a.cpu().double() - b).norm() / b.norm()).item() for a, b in zip(got, want)])
    assert all(sorted_ <= 1.05 * plain for plain, sorted_ in zip(*errors)), errors


@pytest.mark.parametrize("vdt,pdt", [(torch.bfloat16, torch.float32), (torch.float16, torch.float16)])
@pytest.mark.parametrize("D", [16, 32, 48])
def test_positions_that_are_not_finite(D, vdt, pdt, fda_env):
    """NaN and infinite coordinates give NaN gradients where the plain kernel gives them, and nowhere else."""
    shapes, Q, K = [(4, 5, 6), (2, 3, 3)], 60, 4
    value, sh, lsi, packed, grad_out = fda_oracle.make_inputs(shapes, 2, Q, 2, D, K, seed=D, lo=-0.2, hi=1.2)
    nan, inf = float("nan"), float("inf")
    for n, point in enumerate([(nan, 0.4, 0.4), (0.4, inf, 0.4), (0.4, 0.4, -inf), (nan, inf, 0.4), (7.0, nan, 0.4), (nan, nan, nan),
                               (inf, -inf, nan), (6e4, 0.4, -6e4)]):
        packed[n % 2, 7 * n, 1, 3 * n:3 * n + 3] = torch.tensor(point)
    v, pk, go = value.to("cuda", vdt), packed.to("cuda", pdt), grad_out.to("cuda", vdt)
    results = []
    for mode in ("0", "2"):
        fda_env(FDA_BWD_SORT=mode, FDA_BINNING="0")
        results.append(capi.backward(v, sh.cuda(), lsi.cuda(), pk, go, K))
    ulp = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 0.0}
    for a, b, dt in zip(*results, (vdt, pdt)):
        ok = torch.isfinite(a)
        assert torch.equal(ok, torch.isfinite(b)) and not ok.all()
        a, b = a.float()[ok], b.float()[ok]
        assert ((a - b).abs() <= 2 * ulp[dt] * a.abs() + 2e-5 * a.abs().max()).all()   # as in test_walk_matches_oracle, on both sides


@pytest.mark.parametrize("G,D,levels", [(64, 32, 3), (40, 16, 5), (401, 16, 3), (600, 32, 2)])
def test_many_heads(G, D, levels, fda_env):
    """More (level, head) regions than the usual few dozen: 192, 200, and over a thousand, whose tables leave less room for blocks."""
    shapes = [(2, 3, 4), (2, 2, 2), (1, 2, 1), (1, 1, 2), (1, 1, 1)][:levels]
    value, sh, lsi, packed, grad_out = fda_oracle.make_inputs(shapes, 2, 30, G, D, 4, seed=G, lo=-0.3, hi=1.3)
    v, pk, go = value.to("cuda", torch.bfloat16), packed.cuda(), grad_out.to("cuda", torch.bfloat16)
    results = []
    for mode in ("0", "2"):
        fda_env(FDA_BWD_SORT=mode, FDA_BINNING="0")
        assert (capi.backward_path(v, pk, 4) >= 2) == (mode == "2")
        results.append(capi.backward(v, sh.cuda(), lsi.cuda(), pk, go, 4))
    for a, b, ulp in zip(*results, (2.0 ** -8, 0.0)):
        a, b = a.float(), b.float()
        assert ((a - b).abs() <= 2 * ulp * a.abs() + 2e-5 * a.abs().max()).all()   # as in test_walk_matches_oracle, on both sides
