"""Rules that pick a launch by the rows at hand, on both sides of their lines,
against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,bits", [(np.uint16, 16), (np.uint32, 27), (np.uint64, 50)])
@pytest.mark.parametrize("n", [2048, 2049, 4097, 148 * 4 * 2048, 148 * 4 * 2048 + 1])
def test_plain_rounds_by_chunk(ctx, n, dtype, bits):
    """The plain comparator's chunks: one tile while all tiles run at once, two beyond."""
    rng = np.random.default_rng(n)
    bank = rng.integers(0, 1 << bits, size=n, dtype=np.uint64).astype(dtype)
    order, group = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    ng = ctx.sort_round_plain(bank, bits, order, out_group=group)
    o, g, _, ng_ref = O.sort_round(bank)
    assert ng == ng_ref and np.array_equal(order, o) and np.array_equal(group, g)
