"""On-chip sorts of keys that defeat their first bucketings: repeating codes and
one far key, keys of a few low bits and the highest, and keys laid out against
the places the splitters are taken at.  Results against the oracle, and the time
of a segment against that of random keys: a sort that counts through one large
bucket takes 30 to 180 times as long."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TIERS = {256: 32, 512: 64, 1024: 128, 2048: 256, 2304: 256, 4096: 512, 8192: 1024}   # rows: threads


def _splitter_places(rows):
    nt, m = TIERS[rows], np.uint64(0xFFFFFFFF)
    t = np.arange(nt, dtype=np.uint64)
    a, z = t * np.uint64(rows) // np.uint64(nt), (t + np.uint64(1)) * np.uint64(rows) // np.uint64(nt)
    h = ((t + np.uint64(1)) * np.uint64(0x9E3779B9)) & m
    h = ((h ^ (h >> np.uint64(15))) * np.uint64(0x2C1B3C6D)) & m
    return a + (h * (z - a) >> np.uint64(32))


def _segment(kind, rows):
    i = np.arange(rows, dtype=np.uint64)
    if kind == "random":
        return np.random.default_rng(rows).integers(0, 1 << 50, size=rows, dtype=np.uint64)
    if kind == "against":   # every splitter is 0; the other rows a few codes above it
        k = np.uint64(1) + (i * np.uint64(7)) % np.uint64(rows // 2)
        k[_splitter_places(rows)] = 0
        k[int(np.setdiff1d(i, _splitter_places(rows))[0])] = np.uint64(1) << np.uint64(62)
        return k
    if kind == "low bits":
        k = i % np.uint64(8) + ((i * i) << np.uint64(3)) % np.uint64(64)
        k[rows // 3] = np.uint64(1) << np.uint64(63)
        return k
    k = i % np.uint64(int(kind))
    k[rows // 2] = np.uint64(1) << np.uint64(49)
    return k


KINDS = ["8", "24", "1000", "low bits", "against"]


@pytest.mark.parametrize("rows", sorted(TIERS))
@pytest.mark.parametrize("kind", KINDS)
def test_skewed_segments(ctx, kind, rows):
    bank = np.concatenate([_segment(kind, rows), _segment(kind, rows)[:rows - 1], _segment("random", rows)])
    n = bank.shape[0]
    in_group = np.repeat(np.arange(3, dtype=np.uint32), [rows, rows - 1, rows])
    # the same segments as a round after another, and alone in a round
    order, group = np.arange(n, dtype=np.uint32), np.zeros(n, np.uint32)
    ng = ctx.sort_round(bank, 64, order, in_group=in_group, out_group=group)
    o, g, _, ng_ref = O.sort_round(bank, order=np.arange(n, dtype=np.uint32), in_group=in_group)
    assert ng == ng_ref and np.array_equal(order, o) and np.array_equal(group, g)
    bank = bank[:rows]
    order, group = np.zeros(rows, np.uint32), np.zeros(rows, np.uint32)
    ng = ctx.sort_round(bank, 64, order, out_group=group)
    o, g, _, ng_ref = O.sort_round(bank)
    assert ng == ng_ref and np.array_equal(order, o) and np.array_equal(group, g)


@pytest.mark.parametrize("rows", [2048, 4096, 8192])
@pytest.mark.parametrize("kind", KINDS)
def test_skewed_segments_take_no_longer_than_a_network(ctx, kind, rows):
    """At most 10 times the on-chip time of random keys (a network of
    log2(rows)^2 / 2 steps over shared memory is estimated at 2 to 4)."""
    import torch
    segs = 296
    n = rows * segs
    in_group = torch.arange(n, dtype=torch.int32, device="cuda") // rows
    iota = torch.arange(n, dtype=torch.int32, device="cuda")
    group = torch.empty_like(iota)
    best = {}
    for k in ("random", kind):
        bank = torch.from_numpy(np.tile(_segment(k, rows), segs).view(np.int64)).cuda()
        torch.cuda.synchronize()
        times = []
        for _ in range(4):
            order = iota.clone()
            torch.cuda.synchronize()
            ctx.profile(True)
            ctx.sort_round(bank, 64, order, in_group=in_group, out_group=group)
            prof = ctx.profile_report()
            ctx.profile(False)
            times.append(sum(v["ms"] for name, v in prof.items() if name.startswith("block_sort")))
        best[k] = min(times[1:])
    assert 0 < best[kind] < 10 * best["random"], best


@pytest.mark.parametrize("values", [2, 16, 200, 3000])
@pytest.mark.parametrize("zipf", [False, True])
@pytest.mark.parametrize("bits", [50, 60, 64])
def test_few_values(ctx, bits, zipf, values):
    """Segments of every tier whose keys are a few long codes: rows of one key are
    told apart by their positions, beside dropped low bits or next to the key."""
    rng = np.random.default_rng(values + bits)
    codes = rng.integers(0, (1 << bits) - 1, size=values, dtype=np.uint64, endpoint=True)
    codes[1] = codes[0] ^ np.uint64(1)   # the same but for the last bit
    p = 1.0 / np.arange(1, values + 1) if zipf else np.ones(values)
    sizes = [s - d for s in sorted(TIERS) for d in (0, 1, 40)] + [128, 130, 20_000]
    bank = codes[rng.choice(values, size=sum(sizes), p=p / p.sum())]
    in_group = np.repeat(np.arange(len(sizes), dtype=np.uint32), sizes)
    order_in = rng.permutation(bank.shape[0]).astype(np.uint32)
    order, group, keys = order_in.copy(), np.zeros_like(order_in), np.zeros_like(bank)
    ng = ctx.sort_round(bank, bits, order, in_group=in_group, out_group=group, sorted_bank=keys)
    o, g, k, ng_ref = O.sort_round(bank, order=order_in, in_group=in_group)
    assert ng == ng_ref and np.array_equal(order, o) and np.array_equal(group, g) and np.array_equal(keys, k)
