"""Calls that run out of workspace half-way, with the next round's bank already
being stitched on the context's second stream: they say so, and the context's
next call is exact."""
import numpy as np
import pytest

from fastmulticolsort_b200 import capi
from fastmulticolsort_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

BITS, SPLIT = [8, 24, 40], [40, 32]


@pytest.mark.parametrize("how", ["plan", "batch"])
def test_out_of_budget_then_exact(how):
    import torch
    sizes = [150_000, 1, 90_000, 60_001]
    n, few = sum(sizes), 9_001
    cols, bw = W.cols_uniform(n, BITS, seed_index=3, distinct=[9, 2000, 1 << 30])
    dev = [torch.from_numpy(c.view({2: np.int16, 4: np.int32, 8: np.int64}[c.itemsize])).cuda() for c in cols]
    order, group = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()

    def run(ctx, rows):
        part = [d[:rows] for d in dev]
        if how == "plan":
            return ctx.run_plan(part, bw, SPLIT, order[:rows], group[:rows])
        return ctx.run_batch(part, bw, SPLIT, sizes if rows == n else [rows], order[:rows], group[:rows])

    def exact(rows):
        o, g, _ = O.run_plan_sort([c[:rows] for c in cols], bw, SPLIT)
        return (np.array_equal(order[:rows].cpu().numpy().view(np.uint32), o) and
                np.array_equal(group[:rows].cpu().numpy().view(np.uint32), g))

    with capi.Context(0) as ctx:
        run(ctx, few)
        least = ctx.workspace_bytes()
        run(ctx, n)
        most = ctx.workspace_bytes()
    refused = 0
    for k in range(12):   # limits that end the call at one buffer after the other
        with capi.Context(0, least + (most - least) * k // 12) as ctx:
            run(ctx, few)
            try:
                run(ctx, n)
            except capi.FmcsError as e:
                assert e.code == capi.FMCS_E_OOM
                refused += 1
            run(ctx, few)
            assert exact(few), k
    assert refused > 6
