"""Groups whose key bits run out at the first, second or third radix level, of
more rows than a warp copies (4096) and of fewer: plans on both sides of the
row count from which groups are found by flags, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _codes(bits, groups):
    rng = np.random.default_rng(groups)
    if bits <= 16:
        return rng.permutation(1 << bits)[:groups]
    # two codes for each of their first bits: both still in one large segment at the third level
    c = rng.permutation(1 << (bits - 4))[:groups // 2] << 4
    return np.concatenate([c, c + 9])


@pytest.mark.parametrize("rows", [4097, 5000, 8192])
@pytest.mark.parametrize("bits,groups", [(8, 120), (8, 256), (12, 128), (12, 700), (20, 126), (20, 300)])
def test_large_groups(ctx, bits, groups, rows):
    rng = np.random.default_rng(rows)
    v = np.repeat(_codes(bits, groups), rows).astype(np.uint16 if bits <= 16 else np.uint32)
    v = rng.permutation(v)
    n = v.shape[0]
    o, g, ng_ref = O.run_plan_sort([v], [bits], [bits])
    order, group = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    assert ctx.run_plan([v], [bits], [bits], order, group) == ng_ref
    assert np.array_equal(order, o) and np.array_equal(group, g)
    order[:] = 0
    assert ctx.run_plan([v], [bits], [bits], order, None) == ng_ref   # the count alone
    assert np.array_equal(order, o)


@pytest.mark.parametrize("n", [(1 << 20) - 1, 1 << 20, (1 << 20) + 3])
@pytest.mark.parametrize("kind,bits,split", [
    ("few", [9, 5], [14]), ("few", [16, 8], [24]), ("two", [40], [40]), ("skip", [40], [40]),
    ("one_hot", [40], [40]), ("few", [9, 5, 12], [9, 5, 12]), ("one_hot", [40, 9], [40, 9]), ("few", [7, 33], [20, 20])])
def test_flags_and_keys(ctx, kind, bits, split, n):
    """Few values, two values in the highest bit, a first level to skip, one hot
    bucket; one round and several."""
    rng = np.random.default_rng(n + len(kind))
    cols = []
    for w in bits:
        if kind == "two":
            v = rng.integers(0, 2, size=n) << (w - 1)
        elif kind == "skip":
            v = rng.integers(0, 1 << (w - 9), size=n)
        elif kind == "one_hot" and w > 16:
            v = rng.integers(0, 1 << (w - 26), size=n)
            far = rng.random(n) < 0.01
            v[far] = rng.integers(0, 1 << w, size=int(far.sum()))
        else:
            v = rng.permutation(1 << min(w, 16))[:3 + w][rng.integers(0, 3 + w, size=n)]
        cols.append(v.astype(np.uint16 if w <= 16 else np.uint32 if w <= 32 else np.uint64))
    o, g, ng_ref = O.run_plan_sort(cols, bits, split)
    order, group = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    assert ctx.run_plan(cols, bits, split, order, group) == ng_ref
    assert np.array_equal(order, o) and np.array_equal(group, g)


@pytest.mark.parametrize("runs,n", [(2, 100_000), (3, 1_000_002), (8, 20_000), (9, 90_000), (4097, 40_970), (5, 5)])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint64])
def test_hash_ids_in_order(ctx, runs, n, dtype):
    """A hash round that is not the last and whose ids are in order already: one
    value inside every run of the round before, from an arbitrary order."""
    rng = np.random.default_rng(n)
    in_group = np.arange(n, dtype=np.uint32) // np.uint32(runs)
    order_in = rng.permutation(n).astype(np.uint32)
    bank = np.zeros(n, dtype)
    bank[order_in] = rng.integers(0, 200, size=int(in_group[-1]) + 1)[in_group]
    order, group = order_in.copy(), np.zeros(n, np.uint32)
    ng = ctx.hash_round(bank, order, in_group=in_group, out_group=group, last_round=False)
    o, g, _, ng_ref = O.hash_round(bank, order=order_in, in_group=in_group)
    assert ng == ng_ref == in_group[-1] + 1
    assert np.array_equal(order, o) and np.array_equal(group, g)


@pytest.mark.parametrize("n", [300_000, 1_200_000])
def test_hash_plan_dependent_column(ctx, n):
    """GROUP BY over three banks whose second column follows from the first: the
    middle round's ids are in order.  Eager and as a captured graph."""
    import torch
    rng = np.random.default_rng(n)
    a = rng.integers(0, n // 3, size=n).astype(np.uint32)
    cols = [a, (a % np.uint32(251)).astype(np.uint16), rng.integers(0, 4, size=n).astype(np.uint16)]
    bw = split = [22, 8, 2]
    o, g, ng_ref = O.run_plan_hash(cols, bw, split)
    order, group = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    assert ctx.run_plan(cols, bw, split, order, group, hash=True) == ng_ref
    assert np.array_equal(order, o) and np.array_equal(group, g)
    dev = [torch.from_numpy(c.view({2: np.int16, 4: np.int32}[c.itemsize])).cuda() for c in cols]
    d_order, d_group = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    graph = ctx.plan_graph(dev, bw, split, d_order, d_group, hash=True)
    for _ in range(2):
        assert graph.launch() == ng_ref
        assert np.array_equal(d_order.cpu().numpy().view(np.uint32), o)
        assert np.array_equal(d_group.cpu().numpy().view(np.uint32), g)
    graph.close()
