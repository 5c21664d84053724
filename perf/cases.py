"""What this framework is timed at: the calls that its users make, from a few
thousand rows to tens of millions.

A case is a plain dict.  Its ``kind`` says which public entry point carries
it:

  plan    Context.run_plan, a whole ORDER BY (stitch, sort rounds, group ids);
  graph   PlanGraph.launch, the same plan replayed as a CUDA graph;
  hash    Context.run_plan(hash=True), a whole GROUP BY through hash rounds;
  batch   Context.run_batch, many small relations in one call;
  query   a GROUP BY query: plan, the key column in group order, aggregates;
  rounds  stitch + sort_round per bank, a program that drives the rounds itself;
  serve   Server.submit / wait, a burst of requests through the serving loop.

``cols`` lists the columns, one "<bits>:<values>" each, separated by blanks:
<values> is "u" (uniform codes), "z" (Zipf(1.0) codes over min(2^bits, 2^20)
ranks) or a number of distinct codes drawn uniformly.  ``split`` is the plan's
bank widths.  Columns are stored as the reference maps widths to types (up to
16 bits in 2 bytes, up to 32 in 4, else 8) and stay on the device.
"""
import math

import numpy as np
import torch

from fastmulticolsort_b200 import capi

# The bench's table of the reference's experiments (17B33), its Zipf-segmented
# table and its wide table; the instances' columns are its batch's and
# the others are generic.
T_17B33 = "17:8192 33:u"
T_ZIPF = "20:z 24:u 40:u"
T_WIDE = "2:3 1:2 12:2526 12:2526 32:u 7:100"
T_INST = "8:16 24:u 40:u"
T_DIM = "12:2526 7:100"
T_GROUP = "12:2526 33:2000 7:4"
T_MIX = "16:5000 27:u 9:200"


def listed():
    return [
        # The smallest calls: a lookup-sized relation, sorted on its own.
        dict(name="plan_3k", kind="plan", n=3001, cols=T_17B33, split="50"),
        # A page of a larger result, two banks, one column descending.
        dict(name="plan_90k_desc", kind="plan", n=90_001, cols=T_ZIPF, split="64 20", desc="0 1 0"),
        # The reference's own experiment size, sorted column by column.
        dict(name="plan_1m_columns", kind="plan", n=1_048_576, cols=T_17B33, split="17 33"),
        # The headline table through the eager call and through a graph.
        dict(name="plan_16m", kind="plan", n=16_777_216, cols=T_17B33, split="50"),
        dict(name="graph_16m", kind="graph", n=16_777_216, cols=T_17B33, split="50"),
        # A skewed leading column, the largest single table.
        dict(name="plan_zipf_67m", kind="plan", n=67_108_864, cols=T_ZIPF, split="64 20"),
        # ORDER BY over six columns of a wide table.
        dict(name="plan_wide_40m", kind="plan", n=40_000_003, cols=T_WIDE, split="59 7"),
        # GROUP BY through the hash rounds, columns in the planner's order: about
        # five million groups, then four values inside each.
        dict(name="hash_10m", kind="hash", n=10_000_019, cols=T_GROUP, split="45 7", order="1 0 2"),
        # Many relations of very different sizes in one call.
        dict(name="batch_384", kind="batch", instances=384, lo=10, hi=20, cols=T_INST, split="64 8"),
        # A GROUP BY query over two dimension columns: few values, large groups.
        dict(name="query_5m", kind="query", n=5_000_011, cols=T_DIM, split="19"),
        # Rounds driven one by one, on 16- and 32-bit banks.
        dict(name="rounds_4m", kind="rounds", n=4_194_301, cols=T_MIX, split="16 27 9"),
        # A burst of requests of 64 K to 1 M rows at the server.
        dict(name="serve_burst", kind="serve", requests=30, lo=16, hi=20, cols=T_ZIPF),
    ]


MAX_BYTES = 67_108_864 * 24.0   # the largest listed case's inputs and outputs


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _table(rng):
    """Two to five columns of any width; between 20 and 120 bits in all."""
    while True:
        cols = []
        for _ in range(rng.randint(2, 5)):
            w = rng.choice([rng.randint(1, 16), rng.randint(8, 32), rng.randint(20, 48)])
            kind = rng.choice(["u", "u", "z", "d"])
            if kind == "d":
                kind = str(min(1 << w, _log_int(rng, 2, 20_000)))
            cols.append("%d:%s" % (w, kind))
        if 20 <= sum(_bits(" ".join(cols))) <= 120:
            return " ".join(cols)


def _pack(rng, bits):
    """Bank widths over the columns' bits: as wide as they go, one per column,
    or cut anywhere."""
    total = sum(bits)
    how = rng.choice(["wide", "wide", "columns", "cut"])
    if how == "columns" and len(bits) <= 3:
        return " ".join(map(str, bits))
    if how == "cut" and total > 2:
        first = rng.randint(max(1, total - 64), min(64, total - 1)) if total <= 128 else 64
        rest = total - first
        return "%d %d" % (first, rest) if rest <= 64 else "%d 64 %d" % (first, rest - 64)
    out = []
    while total > 0:
        out.append(min(64, total))
        total -= out[-1]
    return " ".join(map(str, out))


def draw(rng):
    kind = rng.choice(["plan", "plan", "plan", "graph", "hash", "batch", "query", "rounds", "serve"])
    cols = rng.choice([T_17B33, T_ZIPF, T_WIDE, T_MIX, None])
    if cols is None:
        cols = _table(rng)
    bits = _bits(cols)
    if kind == "batch":
        lo = rng.randint(6, 14)
        hi = rng.randint(lo + 1, 19)
        return dict(kind=kind, instances=_log_int(rng, 4, 300), lo=lo, hi=hi, cols=T_INST, split="64 8")
    if kind == "serve":
        lo = rng.randint(10, 17)
        return dict(kind=kind, requests=rng.randint(4, 30), lo=lo, hi=rng.randint(lo + 1, 20), cols=rng.choice([T_ZIPF, T_17B33, T_INST]))
    if kind == "query":
        cols = rng.choice([T_DIM, "16:z 9:200", "10:700", "14:z 8:u"])
        bits = _bits(cols)
        return dict(kind=kind, n=_log_int(rng, 5_000, 20_000_000), cols=cols, split=str(sum(bits)))
    if kind == "hash":   # grouping columns: values that repeat
        cols = rng.choice([T_GROUP, T_DIM, "16:z 9:200", "33:5000 7:30", "20:z 24:9000", "40:2000 8:16 30:z"])
        bits = _bits(cols)
    split = " ".join(map(str, bits)) if kind == "rounds" else _pack(rng, bits)
    row = sum(_bytes(b) for b in bits) + 8
    most = MAX_BYTES / row / max(1.0, len(split.split()) / 2.0)
    most = min(most, {"plan": 67_108_864, "graph": 16_777_216, "hash": 16_777_216, "rounds": 16_777_216}[kind])
    case = dict(kind=kind, n=_log_int(rng, 20_000 if kind == "hash" else 1_000, most), cols=cols, split=split)
    if kind == "plan" and rng.random() < 0.3:
        case["desc"] = " ".join(str(rng.randint(0, 1)) for _ in bits)
    return case


def _bits(cols):
    return [int(c.split(":")[0]) for c in cols.split()]


def _bytes(w):
    return 2 if w <= 16 else (4 if w <= 32 else 8)


def _ints(text):
    return [int(x) for x in text.split()]


def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + salt * 7919 + 12345) % (1 << 62))
    return g


def _column(spec, n, seed, salt):
    """n unsigned codes in the reference's storage width, as the signed torch
    type with the same bits."""
    w, values = spec.split(":")
    w = int(w)
    g = _gen(seed, salt)
    if values == "u":
        v = torch.randint(0, 1 << w, (n,), dtype=torch.int64, device="cuda", generator=g)
    else:
        k = min(1 << w, 1 << 20) if values == "z" else min(int(values), 1 << w)
        rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, salt])
        if (1 << w) <= 4 * k:
            codes = rng.permutation(1 << w)[:k]
        else:
            codes = np.unique(rng.integers(0, 1 << w, size=2 * k))
            codes = rng.permutation(codes)[:k]
        codes = torch.from_numpy(codes.astype(np.int64)).cuda()
        k = codes.numel()
        if values == "z":
            cdf = torch.cumsum(torch.arange(1, k + 1, dtype=torch.float64, device="cuda").reciprocal(), 0)
            cdf /= cdf[-1].clone()
            u = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
            pick = torch.searchsorted(cdf, u).clamp_(max=k - 1)
        else:
            pick = torch.randint(0, k, (n,), device="cuda", generator=g)
        v = codes[pick]
    if w > 32:
        return v.contiguous()
    half = 1 << (8 * _bytes(w) - 1)
    v = torch.where(v >= half, v - 2 * half, v)
    return v.to(torch.int16 if w <= 16 else torch.int32).contiguous()


def _columns(cols, n, seed, salt=0):
    return [_column(s, n, seed, salt + k) for k, s in enumerate(cols.split())]


def _sizes(case, count):
    """The relations' row counts: log-uniform, the same for every seed."""
    rng = np.random.default_rng([case["lo"], case["hi"], count])
    return np.floor(2.0 ** rng.uniform(case["lo"], case["hi"], size=count)).astype(np.int64)


def _out(n):
    return torch.zeros(max(n, 1), dtype=torch.int32, device="cuda")[:n]


# One context and one server for the whole program, as its user keeps them.
_kept = {}


def _context():
    if "ctx" not in _kept:
        _kept["ctx"] = capi.Context(torch.cuda.current_device())
    return _kept["ctx"]


def _server():
    if "server" not in _kept:
        _kept["server"] = capi.Server(torch.cuda.current_device(), slots=4)
    return _kept["server"]


def prepare(case, seed):
    kind = case["kind"]
    bw = _bits(case["cols"])
    st = dict(kind=kind, bw=bw)
    if kind == "serve":
        st["server"] = _server()
        st["requests"] = []
        for k, n in enumerate(_sizes(case, case["requests"])):
            n = int(n)
            cols = _columns(case["cols"], n, seed, 100 * (k + 1))
            card = [min(n, 1 << min(w, 20)) for w in bw]
            st["requests"].append((cols, _out(n), _out(n), card))
    else:
        st["ctx"] = _context()
        st["split"] = _ints(case["split"])
        if kind == "batch":
            st["sizes"] = _sizes(case, case["instances"])
            n = int(st["sizes"].sum())
        else:
            n = case["n"]
        st["cols"] = _columns(case["cols"], n, seed)
        st["order"], st["group"] = _out(n), _out(n)
        if case.get("desc"):
            st["desc"] = _ints(case["desc"])
        if case.get("order"):
            st["col_order"] = _ints(case["order"])
        if kind == "query":
            st["payload"] = torch.randint(-(1 << 40), 1 << 40, (n,), dtype=torch.int64, device="cuda", generator=_gen(seed, 55))
            st["key"] = torch.empty_like(st["cols"][0])
            most = min(n, 1 << sum(bw))
            st["agg"] = [torch.zeros(most, dtype=torch.int64, device="cuda") for _ in range(4)]
        if kind == "rounds":
            st["bits"] = st["split"]
            st["banks"] = [torch.zeros(n, dtype={2: torch.int16, 4: torch.int32, 8: torch.int64}[_bytes(w)], device="cuda") for w in st["bits"]]
            st["group2"] = _out(n)
        torch.cuda.synchronize()
        if kind == "graph":
            st["graph"] = st["ctx"].plan_graph(st["cols"], bw, st["split"], st["order"], st["group"])
    torch.cuda.synchronize()
    return st


def run(st):
    kind = st["kind"]
    if kind == "plan":
        ng = st["ctx"].run_plan(st["cols"], st["bw"], st["split"], st["order"], st["group"], descending=st.get("desc"))
        return st["order"], st["group"], ng
    if kind == "graph":
        ng = st["graph"].launch()
        return st["order"], st["group"], ng
    if kind == "hash":
        ng = st["ctx"].run_plan(st["cols"], st["bw"], st["split"], st["order"], st["group"], col_order=st.get("col_order"), hash=True)
        return st["order"], st["group"], ng
    if kind == "batch":
        counts = st["ctx"].run_batch(st["cols"], st["bw"], st["split"], st["sizes"], st["order"], st["group"])
        return st["order"], st["group"], counts.astype(np.int64)
    if kind == "query":
        ctx = st["ctx"]
        ng = ctx.run_plan(st["cols"], st["bw"], st["split"], st["order"], st["group"])
        ctx.gather(st["cols"][0], st["order"], st["key"])
        agg = [a[:ng] for a in st["agg"]]
        ctx.group_aggregate(st["payload"], st["order"], st["group"], ng, *agg, signed=True)
        return [st["order"], st["group"], st["key"], ng] + agg
    if kind == "rounds":
        ctx, prev, ng = st["ctx"], None, 0
        for k, bank in enumerate(st["banks"]):
            ctx.stitch([(st["cols"][k], st["bw"][k], 1, st["bw"][k])], bank)
            out = st["group"] if k % 2 == 0 else st["group2"]
            ng = ctx.sort_round(bank, st["bits"][k], st["order"], in_group=prev, out_group=out)
            prev = out
        return st["order"], prev, ng
    server = st["server"]
    tickets = [server.submit(cols, st["bw"], order, group, cardinality=card) for cols, order, group, card in st["requests"]]
    done = [server.wait(t) for t in tickets]
    out = [x for _, order, group, _ in st["requests"] for x in (order, group)]
    return out + [np.array([d["ngroups"] for d in done], np.int64)]


def work(case):
    """Every column read once, the order and the group vector written once (and
    for a query its payload, its key column's projection and the aggregates)."""
    bits = _bits(case["cols"])
    row = sum(_bytes(w) for w in bits)
    if case["kind"] in ("batch", "serve"):
        n = int(_sizes(case, case.get("instances", case.get("requests"))).sum())
    else:
        n = case["n"]
    total = n * (row + 8.0)
    if case["kind"] == "query":
        total += n * (8.0 + 2 * _bytes(bits[0])) + 32.0 * min(n, 1 << sum(bits))
    return {"bytes": float(total), "flops": 0.0}


def exact(case, seed):
    """Order and group vector of an ORDER BY by plain stable sorts, one column
    after the other from the last; None where numbering is the framework's own
    (hash rounds) or the case is large."""
    if case["kind"] not in ("plan", "graph") or case["n"] > 20_000_000:
        return None
    bits = _bits(case["cols"])
    desc = _ints(case["desc"]) if case.get("desc") else [0] * len(bits)
    cols = []
    for c, w, d in zip(_columns(case["cols"], case["n"], seed), bits, desc):
        v = c.to(torch.int64)
        if w <= 32:
            v &= (1 << (8 * _bytes(w))) - 1
        cols.append((1 << w) - 1 - v if d else v)
    order = torch.arange(case["n"], device="cuda")
    for v in reversed(cols):
        order = order[torch.sort(v[order], stable=True).indices]
    starts = torch.zeros(case["n"], dtype=torch.bool, device="cuda")
    for v in cols:
        s = v[order]
        starts[1:] |= s[1:] != s[:-1]
    group = torch.cumsum(starts.to(torch.int64), 0)
    return order.to(torch.int32), group.to(torch.int32), int(group[-1]) + 1
