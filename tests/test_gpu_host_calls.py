"""What a call asks of the CUDA runtime once its kernels and workspace are warm:
nothing that locks other threads' launches out."""
import numpy as np
import pytest

from fastmulticolsort_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,split", [(3_001, [50]), (60_000, [50]), (1_200_000, [17, 33])])
def test_warm_calls_set_no_kernel_attributes(ctx, n, split):
    import torch
    from torch.profiler import ProfilerActivity, profile
    cols, bw = W.cols_17b33(n, seed_index=5)
    dev = [torch.from_numpy(c.view({4: np.int32, 8: np.int64}[c.itemsize])).cuda() for c in cols]
    order, group = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    for _ in range(2):
        ctx.run_plan(dev, bw, split, order, group)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        ctx.run_plan(dev, bw, split, order, group)
        torch.cuda.synchronize()
    names = [e.name for e in prof.events()]
    assert any("LaunchKernel" in x for x in names)   # runtime calls are recorded
    assert not [x for x in names if "FuncSetAttribute" in x or x in ("cudaMalloc", "cudaFree")]


def test_burst_on_one_host_core():
    """Four server slots whose waits share one core with the submitting thread."""
    import os
    import torch
    from fastmulticolsort_b200 import capi
    from oracle import oracle as O
    allowed = os.sched_getaffinity(0)
    os.sched_setaffinity(0, {min(allowed)})   # threads started from here inherit it
    try:
        with capi.Server(0, slots=4, batch_rows_max=1 << 18) as server:
            runs = []
            for k in range(12):
                cols, bw = W.cols_17b33(20_000 + 30_000 * k, seed_index=k)
                dev = [torch.from_numpy(c.view({4: np.int32, 8: np.int64}[c.itemsize])).cuda() for c in cols]
                order, group = (torch.zeros(cols[0].shape[0], dtype=torch.int32, device="cuda") for _ in range(2))
                runs.append((cols, dev, order, group))
            torch.cuda.synchronize()
            tickets = [server.submit(dev, bw, order, group, split=[17, 33]) for _, dev, order, group in runs]
            for t in tickets:
                assert server.wait(t)["status"] == 0
    finally:
        os.sched_setaffinity(0, allowed)
    for cols, _, order, group in runs:
        o, g, _ = O.run_plan_sort(cols, bw, [17, 33])
        assert np.array_equal(order.cpu().numpy().view(np.uint32), o)
        assert np.array_equal(group.cpu().numpy().view(np.uint32), g)


def test_serving_warm_up_shares_launches():
    """The warm-up leaves the shared launches' workspace grown: it has to make some."""
    import torch
    from fastmulticolsort_b200 import capi, serving
    rng = np.random.default_rng(4)
    pool = []
    for n in rng.integers(60_000, 300_000, size=24):
        cols = [serving._store(torch, serving._uniform_codes(torch, rng, int(n), w), w) for w in (8, 24, 40)]
        pool.append(dict(n=int(n), widths=[8, 24, 40], cols=cols, card=[min(int(n), 1 << w) for w in (8, 24, 40)]))
    with capi.Server(0, slots=4, batch_rows_max=1 << 20) as server:
        assert serving.warm(torch, server, pool, 4) > len(pool) // 4
