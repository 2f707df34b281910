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
