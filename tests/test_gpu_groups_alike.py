"""Batches of cells of one tile and chunk count choose their group size by what
the rounds cost: launches small enough to reach every size (1, 2, 3, 4 and 6
subcarriers), a cap in between, and full groups give the outputs of one
subcarrier a group, bit for bit."""
from __future__ import annotations

import pytest
import torch

from test_gpu_walk import Batch, same

pytestmark = pytest.mark.gpu

CASES = [  # (kind, nAnt, nLayers): exact tiles outside the unrolled kernels, padded tiles, complex half
    ("cf32", 16, 2), ("cf32", 48, 4), ("cf32", 24, 8), ("cf32", 160, 16),
    ("cf32", 20, 1), ("cf32", 33, 3), ("cf32", 40, 12), ("half", 16, 4), ("half", 48, 8),
]


@pytest.mark.parametrize("kind,ant,lay", CASES)
def test_group_size_does_not_change_results(aeq, wl, cuda, kind, ant, lay):
    # 148 warps (one a block, one block an SM): 12, 25, 49 and 74 PRB take groups of 1, 3, 4 and 6 (or 2 and 3)
    for prbs in ((12,), (25,), (49,), (40, 34)):
        b = Batch(aeq, wl, cuda, kind, shapes=[(p, ant, lay, 7 + i, 16) for i, p in enumerate(prbs)])

        def run(cap, warps, ctas):
            descs, outs = b.outputs()
            aeq.pusch_eq_fused(descs, aeq.make_tuning("fp16", warps, ctas, cap))
            torch.cuda.synchronize()
            return outs

        ref = run(1, 4, 1)
        assert all(torch.isfinite(l).all() for l, _ in ref)
        for warps, ctas in ((1, 1), (2, 1), (0, 0)):
            for cap in (0, 3, 32):
                assert same(ref, run(cap, warps, ctas)), (prbs, warps, ctas, cap)
