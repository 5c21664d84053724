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


@pytest.mark.parametrize("nseg", [127, 128, 129, 255, 256, 131, 4 * 256 * 148 + 5])
@pytest.mark.parametrize("kind", ["ones", "one pair last", "pairs", "mixed"])
def test_segments_by_warp(ctx, nseg, kind):
    """The classification's steps of 128 segments a warp: all of one row, one that
    is not, none that are; several rounds of a plan and a batch."""
    rng = np.random.default_rng(nseg)
    sizes = np.ones(nseg, np.int64)
    if kind == "one pair last":
        sizes[-1] = 2
    elif kind == "pairs":
        sizes[:] = 2
    elif kind == "mixed":
        sizes = rng.choice([1, 1, 1, 1, 2, 3, 17, 40], size=nseg)
    n = int(sizes.sum())
    first = rng.permutation(np.repeat(np.arange(nseg), sizes)).astype(np.uint32)
    cols = [first, rng.integers(0, 3, size=n).astype(np.uint16), rng.integers(0, 5, size=n).astype(np.uint16)]
    bw = split = [20, 2, 3]
    o, g, ng_ref = O.run_plan_sort(cols, bw, split)
    order, group = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    assert ctx.run_plan(cols, bw, split, order, group) == ng_ref
    assert np.array_equal(order, o) and np.array_equal(group, g)
    if n > 1000:
        counts = ctx.run_batch(cols, bw, split, [n], order, group)
        assert counts[0] == ng_ref and np.array_equal(order, o) and np.array_equal(group, g)
    # the instances themselves as segments, most of one row
    few = sizes[:3000]
    n = int(few.sum())
    cols = [c[:n].copy() for c in cols[1:]]
    order, group = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    ctx.run_batch(cols, [2, 3], [2, 3], few, order, group)
    off = 0
    for size in few[:300]:
        o, g, _ = O.run_plan_sort([c[off:off + size].copy() for c in cols], [2, 3], [2, 3])
        assert np.array_equal(order[off:off + size], o) and np.array_equal(group[off:off + size], g)
        off += size


@pytest.mark.parametrize("n", [1, 2, 16, 17, 33, 129, 257, 513, 1025, 2049, 2305, 4097, 8192, 8193])
@pytest.mark.parametrize("values", [1, 2, 1 << 20])
def test_small_hash_plans(ctx, n, values):
    """Clustering sorts that fit one tier, one value among them; eager and captured."""
    import torch
    rng = np.random.default_rng(n)
    cols = [rng.integers(0, values, size=n).astype(np.uint32), rng.integers(0, 3, size=n).astype(np.uint16),
            rng.integers(0, 2, size=n).astype(np.uint16)]
    bw = split = [20, 2, 1]
    o, g, ng_ref = O.run_plan_hash(cols, bw, split)
    order, group = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    assert ctx.run_plan(cols, bw, split, order, group, hash=True) == ng_ref
    assert np.array_equal(order, o) and np.array_equal(group, g)
    dev = [torch.from_numpy(c.view({2: np.int16, 4: np.int32}[c.itemsize])).cuda() for c in cols]
    d_order, d_group = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    graph = ctx.plan_graph(dev, bw, split, d_order, d_group, hash=True)
    assert graph.launch() == ng_ref
    assert np.array_equal(d_order.cpu().numpy().view(np.uint32), o)
    assert np.array_equal(d_group.cpu().numpy().view(np.uint32), g)
    graph.close()


@pytest.mark.parametrize("n", [8193, 8193 + 127, 20_001, 300_001, 1_300_003])
@pytest.mark.parametrize("widest", [4, 8])
def test_plans_of_unaligned_columns(ctx, n, widest):
    """Columns and outputs one element off a 16-byte boundary: bank and first-level
    histogram from warps of 128 rows whose last are past the end."""
    import torch
    rng = np.random.default_rng(n)
    bw = [12, 27] + ([40] if widest == 8 else [])
    types = [np.uint16, np.uint32, np.uint64]
    signed = {2: np.int16, 4: np.int32, 8: np.int64}
    cols = [rng.integers(0, 1 << w, size=n, dtype=np.uint64).astype(t) for w, t in zip(bw, types)]
    cols[0] %= 5
    dev = []
    for c in cols:
        d = torch.from_numpy(np.concatenate([c[:1], c]).view(signed[c.itemsize])).cuda()
        dev.append(d[1:])
    order, group = (torch.full((n + 2,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    for split in ([sum(bw)] if sum(bw) <= 64 else [64, sum(bw) - 64], bw):
        o, g, ng_ref = O.run_plan_sort(cols, bw, split)
        assert ctx.run_plan(dev, bw, split, order[1:n + 1], group[1:n + 1]) == ng_ref
        h_order, h_group = order.cpu().numpy(), group.cpu().numpy()
        assert np.array_equal(h_order[1:n + 1].view(np.uint32), o) and np.array_equal(h_group[1:n + 1].view(np.uint32), g)
        assert (h_order[[0, n + 1]] == -7).all() and (h_group[[0, n + 1]] == -7).all()
