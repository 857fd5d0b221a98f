"""How many subcarriers a warp groups changes nothing: every grouping rule's
boundary (one subcarrier a group, as many groups as resident warps, several
rounds, groups handed out dynamically or not) gives the LLRs and Y_eq of the
same cells with one fixed grouping, bit for bit."""
from __future__ import annotations

import pytest
import torch

from test_gpu_walk import Batch, same, walk

pytestmark = pytest.mark.gpu

# Launch shapes set the resident warps: 148 x warps x CTAs per SM on a B200.
SHAPES = [(0, 0), (1, 1), (2, 1), (4, 1)]
CASES = {
    "uniform": [(p, 64, 8, 11, 256) for p in (1, 12, 25)],              # 12, 144, 300 subcarriers
    "uniform_2_layers": [(37, 32, 2, 14, 64)],
    "uniform_16_layers": [(13, 128, 16, 7, 16)],
    "mixed": [(1, 16, 1, 11, 4), (20, 256, 4, 9, 16), (3, 100, 12, 14, 256), (9, 24, 3, 5, 64), (12, 64, 8, 11, 16)],
    "ragged_many": [(1 + i % 5, 8 + 12 * (i % 9), 1 + i % 11, 5 + i % 10, (4, 16, 64, 256)[i % 4]) for i in range(40)],
    "half_mixed": [(20, 256, 4, 9, 16), (3, 32, 16, 14, 256), (31, 16, 2, 5, 64)],
    "half_uniform": [(50, 32, 4, 11, 64)],
}


@pytest.mark.parametrize("prec", ["fp16", "bf16x3"])
@pytest.mark.parametrize("name", CASES)
def test_grouping_does_not_change_results(aeq, wl, cuda, name, prec):
    half = name.startswith("half")
    if half and prec != "fp16":
        pytest.skip("complex-half cells take FP16 operands")
    b = Batch(aeq, wl, cuda, "half" if half else "cf32", shapes=CASES[name])

    def run(tuning):
        descs, outs = b.outputs()
        aeq.pusch_eq_fused(descs, tuning)
        torch.cuda.synchronize()
        return outs

    with walk(static=True):
        ref = run(aeq.make_tuning(prec, 4, 1, 1))
    for l, y in ref:
        assert torch.isfinite(l).all() and torch.isfinite(torch.view_as_real(y) if y.is_complex() else y).all()
    for w, k in SHAPES:
        for cap in (0, 2, 32):
            for static in (False, True):
                with walk(static):
                    assert same(ref, run(aeq.make_tuning(prec, w, k, cap))), (w, k, cap, static)
