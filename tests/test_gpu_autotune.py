"""What the autotuner times is what the cost model adds up: the kernels that a
round of a larger plan launches."""
import pytest

from fastmulticolsort_b200 import autotune

pytestmark = pytest.mark.gpu


def _ran(ctx, call):
    call()
    ctx.profile(True)
    call()
    prof = ctx.profile_report()
    ctx.profile(False)
    return {k for k in prof if not k.startswith("_")}


def test_fixed_cost_of_a_round(ctx):
    """A radix level, a tier and the group ids, as any round has them; not the one
    launch that a small round takes."""
    ran = _ran(ctx, autotune.fixed_round(ctx))
    assert {"classify", "tile_prefix", "msd_hist", "msd_plan", "msd_scatter", "boundary_scan"} <= ran
    assert [k for k in ran if k.startswith(("thread_sort", "warp_sort", "block_sort"))]


@pytest.mark.parametrize("size", [2, 8, 32, 128, 512, 8192])
def test_group_sorts_are_counted(ctx, size):
    """Every kernel between a segmented round's boundary scans is one of the group
    sorts (and the hand-over of the counters)."""
    import torch
    n = 1 << 16
    bank = torch.randint(0, 1 << 15, (n,), dtype=torch.int32, device="cuda")
    in_group = torch.arange(n, dtype=torch.int32, device="cuda") // size
    group = torch.empty_like(bank)
    ran = _ran(ctx, lambda: ctx.sort_round(bank, 15, torch.arange(n, dtype=torch.int32, device="cuda"),
                                           in_group=in_group, out_group=group))
    assert {k for k in ran if not k.startswith(autotune.GROUP_SORT_KERNELS)} <= {"boundary_scan", "publish"}
    assert [k for k in ran if k.startswith(("thread_sort", "warp_sort", "block_sort"))]


@pytest.mark.parametrize("n", [100, 1025, 8192])
def test_small_plans_go_by_their_name(ctx, n):
    """The profiler reports a small plan's one launch as that, not as a tier."""
    import torch
    col = torch.arange(n, dtype=torch.int32, device="cuda")
    order, group = torch.empty_like(col), torch.empty_like(col)
    assert _ran(ctx, lambda: ctx.run_plan([col], [20], [12, 8], order, group)) == {"small_plan"}
