"""The sort engine's branches at the sizes where they can go wrong, bit-exact
against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _segmented(ctx, sizes, bank, key_bits, seed, want_keys=False):
    """One segmented round over segments of these sizes, from an arbitrary
    previous order; compared with the oracle."""
    n = int(np.sum(sizes))
    in_group = np.repeat(np.arange(len(sizes), dtype=np.uint32), sizes)
    order_in = np.random.default_rng(seed).permutation(n).astype(np.uint32)
    order, group = order_in.copy(), np.zeros(n, np.uint32)
    keys = np.zeros(n, bank.dtype) if want_keys else None
    ng = ctx.sort_round(bank, key_bits, order, in_group=in_group, out_group=group, sorted_bank=keys)
    o, g, k, ng_ref = O.sort_round(bank, order=order_in, in_group=in_group)
    assert ng == ng_ref
    assert np.array_equal(order, o)
    assert np.array_equal(group, g)
    if want_keys:
        assert np.array_equal(keys, k)


@pytest.mark.parametrize("want_keys", [False, True])
@pytest.mark.parametrize("dtype,bits", [(np.uint16, 16), (np.uint32, 32), (np.uint64, 64)])
@pytest.mark.parametrize("pattern", [[1], [1, 1, 2], [1, 20, 1, 300, 1], [8191, 1, 1, 9000, 1]])
def test_one_row_segments(ctx, pattern, dtype, bits, want_keys):
    """One-row segments beside longer ones (their keys are written only when
    the caller asks for the sorted bank); keys of an earlier round are left
    in the workspace first."""
    sizes = (pattern * (40000 // sum(pattern) + 1))
    n = int(np.sum(sizes))
    rng = np.random.default_rng(len(sizes))
    stale = np.full(n, 7, dtype)
    ctx.sort_round(stale, bits, np.zeros(n, np.uint32), out_group=np.zeros(n, np.uint32))
    bank = (rng.integers(0, 1 << 16, size=n, dtype=np.uint64) % 5 + 5).astype(dtype)
    _segmented(ctx, sizes, bank, bits, 11, want_keys)
