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
