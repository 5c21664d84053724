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


# segment sizes on both sides of every on-chip capacity (and of the powers of
# two that set the bucket count)
EDGES = [2, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2047,
         2048, 2049, 2304, 2305, 4095, 4096, 4097, 8191, 8192]


def _bank(kind, n, bits, rng):
    top = (1 << bits) - 1
    if kind == "uniform":
        return rng.integers(0, top, size=n, dtype=np.uint64, endpoint=True)
    if kind == "few":        # a handful of values: many equal keys
        return rng.integers(0, 3, size=n, dtype=np.uint64) * np.uint64(top // 2)
    if kind == "skewed":     # one leading code holds most rows, the rest of the key spreads
        lead = bits // 3
        hot = rng.random(n) < 0.9
        lead_code = np.where(hot, 1, rng.integers(0, 1 << lead, size=n, dtype=np.uint64)).astype(np.uint64)
        return (lead_code << np.uint64(bits - lead)) | rng.integers(0, 1 << (bits - lead), size=n, dtype=np.uint64)
    # "ends": differences in the highest and the lowest bit only
    return (rng.integers(0, 2, size=n, dtype=np.uint64) << np.uint64(bits - 1)) | rng.integers(0, 2, size=n,
                                                                                               dtype=np.uint64)


@pytest.mark.parametrize("kind", ["uniform", "few", "skewed", "ends"])
@pytest.mark.parametrize("dtype,bits", [(np.uint16, 16), (np.uint32, 32), (np.uint64, 51), (np.uint64, 52),
                                        (np.uint64, 64)])
def test_onchip_segments(ctx, kind, dtype, bits):
    """Bucketing by digit and by splitters, compounds that fit 64 bits (51 key
    bits and 13 position bits) and that do not."""
    rng = np.random.default_rng(bits + len(kind))
    sizes = [int(s) for s in rng.permutation(EDGES * 2)]
    bank = _bank(kind, int(np.sum(sizes)), bits, rng).astype(dtype)
    _segmented(ctx, sizes, bank, bits, 5, want_keys=True)


@pytest.mark.parametrize("n", EDGES)
@pytest.mark.parametrize("kind", ["skewed", "few"])
def test_onchip_whole_round(ctx, n, kind):
    rng = np.random.default_rng(n)
    bank = _bank(kind, n, 64, rng)
    order, group = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    ng = ctx.sort_round(bank, 64, order, out_group=group)
    o, g, _, ng_ref = O.sort_round(bank)
    assert ng == ng_ref and np.array_equal(order, o) and np.array_equal(group, g)


# Row counts around 32 tiles of 4096 (and 2048) rows, where a segment's chunk
# rows begin to be planned in groups of 32, and a ragged larger one.
LEVEL_SIZES = [65535, 65537, 131071, 131072, 131073, 135168, 135169, 700001]


def _level_keys(kind, n, rng):
    if kind == "uniform":
        return rng.integers(0, 1 << 40, size=n, dtype=np.uint64)
    if kind == "skip":       # the first level's digit is the same in every row: one long segment at the second
        return rng.integers(0, 1 << 31, size=n, dtype=np.uint64)
    if kind == "one_hot":    # nearly every row in one bucket at every level, few equal keys
        k = rng.integers(0, 1 << 14, size=n, dtype=np.uint64)
        far = rng.random(n) < 0.01
        k[far] = rng.integers(0, 1 << 40, size=int(far.sum()), dtype=np.uint64)
        return k
    return rng.integers(0, 2, size=n, dtype=np.uint64) << np.uint64(39)   # "two": no key bits left after one level


@pytest.mark.parametrize("n", LEVEL_SIZES)
@pytest.mark.parametrize("kind", ["uniform", "skip", "one_hot", "two"])
@pytest.mark.parametrize("items", [8, 16])
def test_radix_levels(ctx, n, kind, items):
    """HBM levels whose first histogram the stitch counts (a plan), counts
    itself (a round), and the full-array passes."""
    keys = _level_keys(kind, n, np.random.default_rng(n))
    o, g, _, ng_ref = O.sort_round(keys)
    before = ctx.get_tuning("msd_items")
    ctx.set_tuning("msd_items", items)
    try:
        for how in ("plan", "round", "plain"):
            order, group = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
            if how == "plan":
                ng = ctx.run_plan([keys], [40], [40], order, group)
            elif how == "round":
                ng = ctx.sort_round(keys, 40, order, out_group=group)
            else:
                ng = ctx.sort_round_plain(keys, 40, order, out_group=group)
            assert ng == ng_ref, how
            assert np.array_equal(order, o), how
            assert np.array_equal(group, g), how
    finally:
        ctx.set_tuning("msd_items", before)


def test_radix_levels_many_segments(ctx):
    """Large segments on both sides of 32 chunks beside each other."""
    rng = np.random.default_rng(9)
    sizes = [8193, 131072, 131073, 9000, 300000, 8193, 12289, 262145]
    bank = rng.integers(0, 1 << 34, size=int(np.sum(sizes)), dtype=np.uint64)
    _segmented(ctx, sizes, bank, 40, 3, want_keys=True)


@pytest.mark.parametrize("last", [False, True])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.uint32, np.uint64])
def test_hash_runs_by_size(ctx, dtype, last):
    """Parent runs on both sides of every way of numbering them (a thread up to
    8 rows, a warp up to 32, a CTA up to 2048, the table beyond)."""
    rng = np.random.default_rng(dtype().itemsize)
    sizes = [int(x) for x in rng.permutation([1, 2, 3, 7, 8, 9, 31, 32, 33, 2047, 2048, 2049] * 3)]
    n = int(np.sum(sizes))
    in_group = np.repeat(np.arange(len(sizes), dtype=np.uint32), sizes)
    bank = (rng.integers(0, 5, size=n) * 37).astype(dtype)
    order_in = rng.permutation(n).astype(np.uint32)
    order, group = order_in.copy(), np.zeros(n, np.uint32)
    ng = ctx.hash_round(bank, order, in_group=in_group, out_group=group, last_round=last)
    o, g, ids, ng_ref = O.hash_round(bank, order=order_in, in_group=in_group, last_round=last)
    g = ids if last else g   # the last round leaves the ids at their positions
    assert ng == ng_ref
    assert np.array_equal(order, o)
    assert np.array_equal(group, g)


SMALL = [1, 2, 31, 32, 33, 255, 256, 257, 1023, 1024, 1025, 4095, 4096, 4097, 8191, 8192, 8193]


@pytest.mark.parametrize("n", SMALL)
@pytest.mark.parametrize("split", [[64], [1, 63], [5, 30, 29], [16, 16, 16, 16]])
def test_small_plans(ctx, n, split):
    """Plans around the one-launch limit (8192 rows), with repeated codes,
    a descending column and a captured graph."""
    import torch
    rng = np.random.default_rng(n + len(split))
    bw = [12, 31, 21]
    cols = [(rng.integers(0, 3, size=n) * 1365).astype(np.uint16),
            rng.integers(0, 1 << 31, size=n, dtype=np.uint64).astype(np.uint32) % np.uint32(1 + n // 2),
            rng.integers(0, 1 << 21, size=n, dtype=np.uint64).astype(np.uint32)]
    order, group = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    for desc in (None, [0, 1, 0]):
        ng = ctx.run_plan(cols, bw, split, order, group, descending=desc)
        flip = [np.asarray((1 << w) - 1 - c.astype(np.int64)).astype(c.dtype) if desc and desc[k] else c
                for k, (c, w) in enumerate(zip(cols, bw))]
        o, g, ng_ref = O.run_plan_sort(flip, bw, split)
        assert ng == ng_ref and np.array_equal(order, o) and np.array_equal(group, g)
    dev = [torch.from_numpy(c.view({2: np.int16, 4: np.int32}[c.itemsize])).cuda() for c in cols]
    d_order, d_group = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    graph = ctx.plan_graph(dev, bw, split, d_order, d_group)
    o, g, ng_ref = O.run_plan_sort(cols, bw, split)
    for _ in range(2):
        assert graph.launch() == ng_ref
        assert np.array_equal(d_order.cpu().numpy().view(np.uint32), o)
        assert np.array_equal(d_group.cpu().numpy().view(np.uint32), g)
    graph.close()


@pytest.mark.parametrize("n", SMALL)
@pytest.mark.parametrize("dtype,bits", [(np.uint16, 9), (np.uint32, 32), (np.uint64, 64)])
def test_small_segmented_rounds(ctx, n, dtype, bits):
    """Segmented rounds around the same limit; a previous order that is not
    ascending inside its segments."""
    rng = np.random.default_rng(n)
    cuts = np.sort(rng.choice(np.arange(1, n), size=min(n - 1, n // 3), replace=False)) if n > 1 else np.array([], int)
    sizes = np.diff(np.concatenate([[0], cuts, [n]]))
    bank = (rng.integers(0, 1 << 9, size=n, dtype=np.uint64) % np.uint64(7)).astype(dtype)
    _segmented(ctx, sizes, bank, bits, n, want_keys=True)
    _segmented(ctx, [n], bank, bits, n)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 4096, 4099, 20001])
@pytest.mark.parametrize("bank_bytes", [1, 2, 4, 8])
@pytest.mark.parametrize("offset", [0, 1])
def test_stitch_slices(ctx, n, bank_bytes, offset):
    """Slices of every source width at every place of the bank (inside a word,
    across its middle, past its end), on and off a 16-byte boundary, rows that
    do not fill a group of four."""
    import torch
    rng = np.random.default_rng(n * 10 + bank_bytes)
    tt = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}
    nt = {1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}
    for widest in (1, 2, 4, 8):
        slices, dev = [], []
        for _ in range(int(rng.integers(1, 8))):
            b = int(rng.choice([x for x in (1, 2, 4, 8) if x <= widest]))
            bits = int(rng.integers(1, 8 * b + 1))
            start = int(rng.integers(1, bits + 1))
            end = int(rng.integers(start, bits + 1))
            v = rng.integers(0, (1 << bits) - 1, size=n, dtype=np.uint64, endpoint=True).astype(nt[b])
            d = torch.zeros(n + 16, dtype=tt[b], device="cuda")
            raw = torch.from_numpy(v.view({1: np.uint8, 2: np.int16, 4: np.int32, 8: np.int64}[b]))
            d[offset:offset + n] = raw.cuda()
            slices.append((v, bits, start, end))
            dev.append((d[offset:offset + n], bits, start, end))
        bank = torch.zeros(n, dtype=tt[bank_bytes], device="cuda")
        torch.cuda.synchronize()
        ctx.stitch(dev, bank)
        want = np.zeros(n, np.uint64)
        for v, bits, start, end in slices:   # shift left by each slice's width, then or it in
            w = end - start + 1
            x = (v.astype(np.uint64) >> np.uint64(bits - end)) & np.uint64((1 << w) - 1)
            want = x if w == 64 else (want << np.uint64(w)) | x
        assert np.array_equal(bank.cpu().numpy().view(nt[bank_bytes]), want.astype(nt[bank_bytes]))
