"""Performance cases of the query-execution core: what is timed, on which inputs, and what it must return.

Each case is a dict of plain values; `kind` picks one of the paths below.  prepare() makes what a user's
program holds before the call (tables resident in device memory, compiled plans, prepared queries),
run() makes one pass through the public entry points, exact() gives the same results in plain torch /
numpy at 64 bits, work() the bytes a pass cannot do without.

  prepared   a prepared query (one CUDA graph) on a small table: a dashboard's or a lookup's query
             repeated with its constants; latency counts.  Hash GROUP BY, delivered in pinned memory.
  burst      a burst of arrived queries of one plan over tables of different size as one prepared group
             (the serving loop's form).
  query      one ad-hoc filter + hash GROUP BY in the engine's sequence of calls (create, batches, run,
             overflow check, fetch), one or two keys.
  pricing    the pricing summary: scan + filter + GROUP BY two 1-byte flags (6 groups), exact sums, the
             headline configuration at 60,000,000 rows; delivered by the one-sync fetch.
  scan       filter + aggregates without GROUP BY over the engine's encoded segment columns (frame of
             reference, double dictionary, decimals), NULLs and deleted rows.
  dense      GROUP BY a small-range integer key (stores, products): 64 groups to hundreds of thousands.
  hicard     GROUP BY a sparse 64-bit key with Zipf skew (users, URLs), results left on the device and
             put in key order (ORDER BY key).
  select     filter -> row indices -> gathers of raw and encoded columns (materialisation of a scan).
  join       filter the build side, join, gather the joined columns, dense GROUP BY: inner over
             consecutive keys (orders x line items) or sparse keys, or LEFT JOIN.
  orderby    expression + sort permutation + gathers (ORDER BY an expression DESC, a date).
  encode     one segment's columns into the stored formats (the flush path).

Tables are cut into segments of 2^20 rows as the engine stores them; row counts are mostly odd, so the
last segment is ragged.
"""
import ctypes

import numpy as np
import torch

from warpstore_b200 import abi, estimator, ops
from warpstore_b200 import query as q
from warpstore_b200 import workloads as W

SEG = W.SEG_ROWS


def listed():
    return [
        # the smallest call: one prepared query over a small table; launches and latency are what it costs
        {"name": "prepared_20k", "kind": "prepared", "rows": 20_000, "groups": 16},
        # eight arrived queries of one plan, tables of 2.5M rows down to 312,500
        {"name": "burst_8x2m", "kind": "burst", "rows": 2_500_000, "groups": 100, "queries": 8},
        # the benchmark's filter + GROUP BY over one segment in the engine's call sequence
        {"name": "query_1m", "kind": "query", "rows": 1 << 20, "groups": 16, "keys": 1},
        # the headline scan
        {"name": "pricing_60m", "kind": "pricing", "rows": W.PRICING_ROWS},
        # a selective revenue scan over encoded columns with NULLs and deleted rows
        {"name": "scan_encoded_30m", "kind": "scan", "rows": 30_000_001, "deleted": True, "percent": 20},
        # totals per store: too many groups for private rows, few enough for shared memory
        {"name": "dense_1500g_16m", "kind": "dense", "rows": 16_777_259, "groups": 1500},
        # the largest: high-cardinality GROUP BY with skew, ORDER BY key
        {"name": "hicard_100m", "kind": "hicard", "rows": W.HC_ROWS, "ranks": W.HC_RANKS},
        # materialise a quarter of a 20M-row table
        {"name": "select_20m", "kind": "select", "rows": 20_000_003, "percent": 25, "deleted": False},
        # the join benchmark: 15M orders (half pass the filter) x 60M line items, 2^20 groups
        {"name": "join_15m_60m", "kind": "join", "build": W.JOIN_BUILD_ROWS, "probe": W.JOIN_PROBE_ROWS,
         "groups": W.JOIN_GROUP_KEYS, "sparse": False, "left": False},
        # LEFT JOIN on sparse keys (hash table), a dimension of 2M rows
        {"name": "leftjoin_2m_12m", "kind": "join", "build": 2_000_003, "probe": 12_000_017, "groups": 5000,
         "sparse": True, "left": True},
        # ORDER BY revenue DESC, date over 4M rows
        {"name": "orderby_4m", "kind": "orderby", "rows": 4_000_037},
        # flush of one full segment: five columns
        {"name": "encode_segment", "kind": "encode", "rows": SEG},
    ]


def _log(rng, lo, hi):
    """An odd-ish size, uniform over the logarithm of [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def _grouped(rng, case, lo, hi, rows):
    """The case with a number of groups that leaves each at least 64 rows (none is empty, whatever the seed)."""
    case["groups"] = _log(rng, min(lo, max(1, case[rows] // 64)), min(hi, max(1, case[rows] // 64)))
    return case


def draw(rng):
    kind = rng.choice(["prepared", "burst", "query", "pricing", "scan", "dense", "hicard", "select", "join",
                       "orderby", "encode"])
    if kind == "prepared":
        return _grouped(rng, {"kind": kind, "rows": _log(rng, 1000, 1_000_000)}, 2, 2000, "rows")
    if kind == "burst":
        return _grouped(rng, {"kind": kind, "rows": _log(rng, 20_000, 2_500_000), "queries": rng.randint(2, 10)}, 4,
                        150, "rows")
    if kind == "query":
        return _grouped(rng, {"kind": kind, "rows": _log(rng, 5000, 8_000_000), "keys": rng.choice([1, 2])}, 2,
                        100_000, "rows")
    if kind == "pricing":
        return {"kind": kind, "rows": _log(rng, 500_000, 60_000_000)}
    if kind == "scan":
        return {"kind": kind, "rows": _log(rng, 100_000, 40_000_000), "deleted": rng.random() < 0.5,
                "percent": _log(rng, 4, 90)}
    if kind == "dense":
        return _grouped(rng, {"kind": kind, "rows": _log(rng, 200_000, 20_000_000)}, 64, 1 << 20, "rows")
    if kind == "hicard":
        return {"kind": kind, "rows": _log(rng, 2_000_000, 60_000_000), "ranks": _log(rng, 100_000, 8_000_000)}
    if kind == "select":
        return {"kind": kind, "rows": _log(rng, 50_000, 30_000_000), "percent": _log(rng, 1, 95),
                "deleted": rng.random() < 0.5}
    if kind == "join":
        build = _log(rng, 50_000, 8_000_000)
        return _grouped(rng, {"kind": kind, "build": build, "probe": build * rng.randint(1, 6) + rng.randint(0, 999),
                              "sparse": rng.random() < 0.5, "left": rng.random() < 0.4}, 64, 1 << 20, "probe")
    if kind == "orderby":
        return {"kind": kind, "rows": _log(rng, 10_000, 6_000_000)}
    return {"kind": kind, "rows": _log(rng, 30_000, SEG)}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _ints(g, lo, hi, n, dtype=torch.int64):
    return torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=dtype)


def _f64(g, n):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _mix(x):
    """A bijection of 52-bit integers (odd multiply, xor-shifts): sparse keys that doubles hold exactly."""
    m = (1 << 52) - 1
    x = (x * 0x5DEECE66D1B5) & m
    x = x ^ (x >> 23)
    x = (x * 0x2545F4914F6D) & m
    return x ^ (x >> 27)


def _segs(n):
    return [min(SEG, n - s) for s in range(0, n, SEG)]


class _Raw:
    """A raw column: views into one tensor."""

    def __init__(self, t, x):
        self.t, self.enc, self.x = t, 0, x

    def view(self, s):
        return abi.ColView(self.x.data_ptr() + s * SEG * self.x.element_size(), self.t, 0, 0, 0)


class _Enc:
    """An encoded column in the engine's segment layout: 16-byte header (int64 base, double 10^s), the
    dictionary of enc 4, codes, 16 pad bytes; one aligned region per segment."""

    def __init__(self, t, enc, codes, base=0, p10=1.0, dictionary=None):
        self.t, self.enc = t, enc
        width = {1: 1, 2: 2, 3: 4, 4: 1, 5: 2, 6: 4}[enc]
        codes = codes.to({1: torch.uint8, 2: torch.int16, 4: torch.int32}[width])
        head = np.zeros(16 + (2048 if enc == 4 else 0), dtype=np.uint8)
        head[:8] = np.frombuffer(np.int64(base).tobytes(), np.uint8)
        head[8:16] = np.frombuffer(np.float64(p10).tobytes(), np.uint8)
        if enc == 4:
            d = np.zeros(256)
            d[:len(dictionary)] = dictionary
            head[16:] = np.frombuffer(d.tobytes(), np.uint8)
        n = codes.numel()
        lens = _segs(n)
        self.stride = (head.size + max(lens) * width + 16 + 255) // 256 * 256
        self.x = torch.zeros((len(lens), self.stride), dtype=torch.uint8, device="cuda")
        self.x[:, :head.size] = torch.from_numpy(head).cuda()
        raw = codes.view(torch.uint8)
        for s, m in enumerate(lens):
            self.x[s, head.size:head.size + m * width] = raw[s * SEG * width:(s * SEG + m) * width]

    def view(self, s):
        return abi.ColView(self.x.data_ptr() + s * self.stride, self.t, 0, self.enc, 0)


def _batches(cols, n, deleted=None):
    """[(rows, deleted bitmap, views)] per segment."""
    return [(m, deleted.data_ptr() + s * (SEG // 8) if deleted is not None else 0, [c.view(s) for c in cols])
            for s, m in enumerate(_segs(n))]


def _env(cols):
    e = q.Env()
    for c in cols:
        e.column(c.t, 0, c.enc)
    return e


def _pack_bits(mask):
    n = mask.numel()
    m = torch.zeros((n + 31) // 32 * 32, dtype=torch.int64, device="cuda")
    m[:n] = mask
    return (m.view(-1, 32) << torch.arange(32, device="cuda")).sum(1).to(torch.int32)


def _jit(e, plan, fn):
    ops.jit_set_mode(abi.JIT_SYNC)
    try:
        return ops.jit_get(e.env, e.ncols, plan, fn, "perf")
    finally:
        ops.jit_set_mode(-1)


def _add(agg, e, arrays):
    ops.check(ops.lib().ws_agg_add_batches(agg.h, e.ncols, *arrays[:4]))


def _pow2(n, least=1024):
    c = least
    while c < n:
        c <<= 1
    return c


def _columns(aq, keys, exact):
    """The result columns of fetched groups: keys, then each aggregate (integer SUM as its two int128
    words, AVG as the quotient)."""
    out = {}
    for k in range(aq.plan.nkeys):
        col = np.ascontiguousarray(keys[:, k])
        out["key%d" % k] = col.view(np.int64) if aq.plan.keyInt[k] else col
    for i, a in enumerate(aq.aggs):
        w = exact[:, a.slot, :]
        cnt = exact[:, a.cnt_slot, 0]
        is_int = bool(aq.plan.aggInt[a.slot]) or a.fn == "COUNT"
        if a.fn == "COUNT":
            v = cnt
        elif a.fn == "AVG":
            v = (w[:, 0] if is_int else np.ascontiguousarray(w[:, 0]).view(np.float64)) / cnt
        elif not is_int:
            v = np.ascontiguousarray(w[:, 0]).view(np.float64)
        else:
            v = w if a.fn == "SUM" else w[:, 0]
        out["%s%d" % (a.fn.lower(), i)] = v
    return out


def _ordered(aq, keys, exact):
    """_columns in key order (a hash GROUP BY delivers its groups in no order)."""
    order = np.lexsort(keys.view(np.int64).T[::-1])
    return _columns(aq, keys[order], exact[order])


def _wide(x):
    """int64 sums as the two words of an int128."""
    x = x.cpu().numpy().astype(np.int64)
    return np.stack([x, x >> 63], axis=1)


def _sum_by(idx, v, n):
    return torch.zeros(n, dtype=v.dtype, device="cuda").scatter_add_(0, idx, v)


def _min_by(idx, v, n, how="amin"):
    start = torch.iinfo(v.dtype).max if how == "amin" else torch.iinfo(v.dtype).min
    return torch.full((n,), start, dtype=v.dtype, device="cuda").scatter_reduce_(0, idx, v, how)


# ---------------------------------------------------------------- filter + GROUP BY (prepared, burst, query)
def _facts(rows, groups, keys, seed):
    """k (and k2): group keys, v int64, f double."""
    g = _gen(seed)
    if keys == 2:
        k2n = max(1, int(groups ** 0.5))
        k = _ints(g, 0, max(1, groups // k2n), rows, torch.int32)
        k2 = _ints(g, 19_000, 19_000 + k2n, rows, torch.int32)
    else:
        k, k2 = _ints(g, 0, groups, rows, torch.int32), None
    return k, k2, _ints(g, 0, 1_000_000, rows), _f64(g, rows)


def _facts_query(keys, cut, enc=None):
    e = q.Env()
    for t in (abi.T_I32, abi.T_I64, abi.T_F64) + ((abi.T_I32,) if keys == 2 else ()):
        e.column(t)
    aggs = [q.Agg("COUNT"), q.Agg("SUM", q.col(1), "BIGINT", True), q.Agg("MIN", q.col(1), "BIGINT", True),
            q.Agg("MAX", q.col(1), "BIGINT", True), q.Agg("AVG", q.col(2), "DOUBLE", True)]
    ks = [(q.col(0), True)] + ([(q.col(3), True)] if keys == 2 else [])
    return e, q.AggQuery(e, q.col(1).lt(cut), ks, aggs)


def _facts_cols(k, k2, v, f):
    return [_Raw(abi.T_I32, k), _Raw(abi.T_I64, v), _Raw(abi.T_F64, f)] + ([_Raw(abi.T_I32, k2)] if k2 is not None
                                                                          else [])


def _facts_exact(k, k2, v, f, cut):
    live = v < cut
    key = k.long() if k2 is None else k.long() * (1 << 32) + k2.long()
    keys, inv = torch.unique(key[live], return_inverse=True)
    n, v, f = keys.numel(), v[live], f[live]
    cnt = _sum_by(inv, torch.ones_like(v), n)
    out = {"key0": (keys if k2 is None else keys >> 32).cpu().numpy()}
    if k2 is not None:
        out["key1"] = (keys & 0xFFFFFFFF).cpu().numpy()
    out.update({"count0": cnt.cpu().numpy(), "sum1": _wide(_sum_by(inv, v, n)), "min2": _min_by(inv, v, n).cpu().numpy(),
                "max3": _min_by(inv, v, n, "amax").cpu().numpy(), "avg4": (_sum_by(inv, f, n) / cnt).cpu().numpy()})
    return out


CUT = 500_000  # half of the rows pass


def _burst_sizes(case):
    return [max(1, case["rows"] // (i + 1)) for i in range(case["queries"])]


def _burst_cut(i):
    return CUT + 40_000 * i  # every query of the burst has its own constant


def _executor(rows, groups, cut, seed):
    cols = _facts_cols(*_facts(rows, groups, 1, seed))
    e, aq = _facts_query(1, cut)
    prog = _jit(e, aq.plan, abi.JF_GROUPED)
    ex = ops.Executor(aq.plan, _pow2(2 * groups), None, e.env, e.ncols, estimator.batch_arrays(_batches(cols, rows)),
                      prog, groups)
    return {"cols": cols, "e": e, "aq": aq, "prog": prog}, ex


def prepare_prepared(case, seed):
    s, s["ex"] = _executor(case["rows"], case["groups"], CUT, seed)
    return s


def run_prepared(s):
    s["ex"].run(s["e"].env)
    ops.sync()
    keys, exact, st = s["ex"].results()
    if st["overflow"] or st["error"]:
        raise RuntimeError("prepared query failed: %s" % st)
    return _ordered(s["aq"], keys, exact)


def exact_prepared(case, seed):
    return _facts_exact(*_facts(case["rows"], case["groups"], 1, seed), CUT)


def prepare_burst(case, seed):
    parts, exs = zip(*[_executor(n, case["groups"], _burst_cut(i), seed * 100 + i)
                       for i, n in enumerate(_burst_sizes(case))])
    return {"parts": parts, "group": ops.ExecGroup(list(exs), parts[0]["prog"])}


def run_burst(s):
    s["group"].run([p["e"].env for p in s["parts"]])
    ops.sync()
    out = []
    for p, ex in zip(s["parts"], s["group"].executors):
        keys, exact, st = ex.results()
        if st["overflow"] or st["error"]:
            raise RuntimeError("prepared query failed: %s" % st)
        out.append(_ordered(p["aq"], keys, exact))
    return out


def exact_burst(case, seed):
    return [_facts_exact(*_facts(n, case["groups"], 1, seed * 100 + i), _burst_cut(i))
            for i, n in enumerate(_burst_sizes(case))]


def prepare_query(case, seed):
    cols = _facts_cols(*_facts(case["rows"], case["groups"], case["keys"], seed))
    e, aq = _facts_query(case["keys"], CUT)
    return {"cols": cols, "e": e, "aq": aq, "prog": _jit(e, aq.plan, abi.JF_GROUPED),
            "cap": W.plain_capacity(aq.plan, case["groups"]),
            "arrays": estimator.batch_arrays(_batches(cols, case["rows"]))}


def run_query(s):
    agg = ops.GpuAggregator(s["aq"].plan, s["cap"])
    _add(agg, s["e"], s["arrays"])
    agg.run(s["e"].env, s["prog"])
    if agg.overflowed():
        raise RuntimeError("hash table overflow")
    keys, _, exact = agg.fetch()
    agg.close()
    return _ordered(s["aq"], keys, exact)


def exact_query(case, seed):
    return _facts_exact(*_facts(case["rows"], case["groups"], case["keys"], seed), CUT)


# ---------------------------------------------------------------- pricing summary
def _pricing(rows, seed):
    g = _gen(seed)
    return [_ints(g, 0, 2557, rows, torch.int32), _ints(g, 1, 51, rows), _ints(g, 90_000, 10_500_001, rows),
            _ints(g, 0, 11, rows), _ints(g, 0, 9, rows), _ints(g, 0, 3, rows, torch.uint8),
            _ints(g, 0, 2, rows, torch.uint8)]


PRICING_CUT = 2467


def prepare_pricing(case, seed):
    x = _pricing(case["rows"], seed)
    cols = [_Raw(abi.T_I32, x[0])] + [_Raw(abi.T_I64, c) for c in x[1:5]] + [_Enc(abi.T_I32, 1, c) for c in x[5:]]
    e = _env(cols)
    ship, qty, price, disc, tax, f1, f2 = (q.col(i) for i in range(7))
    dp = price * (q.ilit(100) - disc)
    aggs = [q.Agg("COUNT"), q.Agg("SUM", qty, "BIGINT", True), q.Agg("SUM", price, "BIGINT", True),
            q.Agg("SUM", dp, "BIGINT", False), q.Agg("SUM", dp * (q.ilit(100) + tax), "BIGINT", False),
            q.Agg("AVG", qty, "BIGINT", True), q.Agg("AVG", price, "BIGINT", True), q.Agg("AVG", disc, "BIGINT", True)]
    aq = q.AggQuery(e, ship.le(PRICING_CUT), [(f1, True), (f2, True)], aggs)
    ds = q.dense_spec(aq.plan, [(0, 2), (0, 1)], case["rows"])
    return {"cols": cols, "e": e, "aq": aq, "ds": ds, "prog": _jit(e, aq.plan, abi.JF_DENSE),
            "arrays": estimator.batch_arrays(_batches(cols, case["rows"])),
            "keys": ops.HostBuffer((6, 2), np.float64), "exact": ops.HostBuffer((6, aq.plan.naggs, 2), np.int64),
            "status": ops.HostBuffer(1, ops.FETCH_STATUS)}


def run_pricing(s):
    agg = ops.GpuAggregator(s["aq"].plan, 1024, s["ds"])
    _add(agg, s["e"], s["arrays"])
    agg.run(s["e"].env, s["prog"])
    agg.fetch_async(6, s["keys"], s["exact"], s["status"])
    ops.sync()
    st = s["status"].array[0]
    if st["overflow"] or st["error"]:
        raise RuntimeError("query failed: %s" % st)
    g = int(st["groups"])
    agg.close()
    return _columns(s["aq"], s["keys"].array[:g], s["exact"].array[:g])


def exact_pricing(case, seed):
    ship, qty, price, disc, tax, f1, f2 = _pricing(case["rows"], seed)
    gi = torch.where(ship <= PRICING_CUT, f1.long() + 3 * f2.long(), 6)  # group 6: rows that fail the filter

    def total(v):
        return _sum_by(gi, v, 7)[:6]
    cnt = total(torch.ones_like(qty))
    have = cnt > 0
    dp = price * (100 - disc)
    sums = [total(v) for v in (qty, price, dp, dp * (100 + tax))]
    avgs = [total(v).double() / cnt for v in (qty, price, disc)]
    out = {"key0": (torch.arange(6, device="cuda") % 3)[have].cpu().numpy(),
           "key1": (torch.arange(6, device="cuda") // 3)[have].cpu().numpy(), "count0": cnt[have].cpu().numpy()}
    for i, v in enumerate(sums):
        out["sum%d" % (i + 1)] = _wide(v[have])
    for i, v in enumerate(avgs):
        out["avg%d" % (i + 5)] = v[have].cpu().numpy()
    return out


# ---------------------------------------------------------------- scan without GROUP BY over encoded columns
DISCOUNTS = [i / 100 for i in range(11)]


def _scan(rows, seed):
    g = _gen(seed)
    ship = _ints(g, 0, 2557, rows, torch.int32)
    qty = _ints(g, 0, 50, rows, torch.uint8)
    price = _ints(g, 90_000, 10_500_001, rows)
    price[_f64(g, rows) < 0.02] = abi.NULL_I64
    disc = _ints(g, 0, 11, rows, torch.uint8)
    tax = _ints(g, 0, 900, rows, torch.int32)
    dead = _f64(g, rows) < 0.03
    return ship, qty, price, disc, tax, dead


def _scan_days(case):
    return max(1, 2557 * case["percent"] // 100)


def prepare_scan(case, seed):
    ship, qty, price, disc, tax, dead = _scan(case["rows"], seed)
    cols = [_Enc(abi.T_I32, 2, ship, base=8000), _Enc(abi.T_I64, 1, qty, base=1), _Raw(abi.T_I64N, price),
            _Enc(abi.T_F64, 4, disc, dictionary=DISCOUNTS), _Enc(abi.T_F64, 5, tax, p10=100.0)]
    e = _env(cols)
    cs, cq, cp, cd, ct = (q.col(i) for i in range(5))
    where = q.and_(q.and_(cs.ge(8100), cs.lt(8100 + _scan_days(case))), q.and_(cd.ge(0.015), cq.lt(40)))
    aggs = [q.Agg("COUNT"), q.Agg("SUM", cp, "BIGINT", True, nullable=True),
            q.Agg("SUM", cp * cd, "DOUBLE", False, nullable=True), q.Agg("MIN", cp, "BIGINT", True, nullable=True),
            q.Agg("MAX", cs, "INT", True), q.Agg("AVG", ct, "DOUBLE", True), q.Agg("SUM", cq, "BIGINT", True)]
    aq = q.AggQuery(e, where, [], aggs)
    dele = _pack_bits(dead) if case["deleted"] else None
    return {"cols": cols, "dele": dele, "e": e, "aq": aq, "prog": _jit(e, aq.plan, abi.JF_NOKEYS),
            "arrays": estimator.batch_arrays(_batches(cols, case["rows"], dele))}


def run_scan(s):
    agg = ops.GpuAggregator(s["aq"].plan, 1)
    _add(agg, s["e"], s["arrays"])
    agg.run(s["e"].env, s["prog"])
    keys, _, exact = agg.fetch()
    agg.close()
    return _columns(s["aq"], keys, exact)


def exact_scan(case, seed):
    ship, qty, price, disc, tax, dead = _scan(case["rows"], seed)
    live = (ship >= 100) & (ship < 100 + _scan_days(case)) & (disc >= 2) & (qty < 39)
    if case["deleted"]:
        live &= ~dead
    some = live & (price != abi.NULL_I64)
    d = torch.tensor(DISCOUNTS, dtype=torch.float64, device="cuda")[disc[some].long()]
    p = price[some]
    t = (tax[live].double() / 100.0).sum() / live.sum()
    one = lambda v: np.array([v.item()])  # noqa: E731
    return {"count0": one(live.sum()), "sum1": _wide(p.sum().view(1)), "sum2": one((p.double() * d).sum()),
            "min3": one(p.min()), "max4": one(ship[live].max().long() + 8000), "avg5": one(t),
            "sum6": _wide((qty[live].long() + 1).sum().view(1))}


# ---------------------------------------------------------------- GROUP BY a small-range key
def _dense(rows, groups, seed):
    g = _gen(seed)
    return (_ints(g, 100, 100 + groups, rows, torch.int32), _ints(g, -5000, 1_000_000, rows),
            _ints(g, 8000, 10557, rows, torch.int32), _f64(g, rows))


def prepare_dense(case, seed):
    k, v, d, f = _dense(case["rows"], case["groups"], seed)
    cols = [_Raw(abi.T_I32, k), _Raw(abi.T_I64, v), _Raw(abi.T_I32, d), _Raw(abi.T_F64, f)]
    e = _env(cols)
    aggs = [q.Agg("COUNT"), q.Agg("SUM", q.col(1), "BIGINT", True), q.Agg("MIN", q.col(1), "BIGINT", True),
            q.Agg("MAX", q.col(2), "INT", True), q.Agg("SUM", q.col(3), "DOUBLE", True)]
    aq = q.AggQuery(e, q.col(2).lt(10_000), [(q.col(0), True)], aggs)
    ds = q.dense_spec(aq.plan, [(100, 99 + case["groups"])], case["rows"])
    prog = _jit(e, aq.plan, abi.JF_GROUPED if ds is None else abi.JF_DENSE)
    return {"cols": cols, "e": e, "aq": aq, "ds": ds, "prog": prog,
            "cap": W.plain_capacity(aq.plan, case["groups"]),
            "arrays": estimator.batch_arrays(_batches(cols, case["rows"]))}


def run_dense(s):
    agg = ops.GpuAggregator(s["aq"].plan, s["cap"], s["ds"])
    _add(agg, s["e"], s["arrays"])
    agg.run(s["e"].env, s["prog"])
    if agg.overflowed():
        raise RuntimeError("hash table overflow")
    keys, _, exact = agg.fetch()
    agg.close()
    return _columns(s["aq"], keys, exact) if s["ds"] is not None else _ordered(s["aq"], keys, exact)


def exact_dense(case, seed):
    k, v, d, f = _dense(case["rows"], case["groups"], seed)
    live = d < 10_000
    keys, inv = torch.unique(k[live].long(), return_inverse=True)
    n, v, d, f = keys.numel(), v[live], d[live].long(), f[live]
    return {"key0": keys.cpu().numpy(), "count0": _sum_by(inv, torch.ones_like(v), n).cpu().numpy(),
            "sum1": _wide(_sum_by(inv, v, n)), "min2": _min_by(inv, v, n).cpu().numpy(),
            "max3": _min_by(inv, d, n, "amax").cpu().numpy(), "sum4": _sum_by(inv, f, n).cpu().numpy()}


# ---------------------------------------------------------------- high-cardinality GROUP BY, ORDER BY key
def _hicard(rows, ranks, seed):
    """Every row's rank is a stratified draw of a bounded power law (the inverse CDF at (i + 0.5) / rows), and
    a fixed 6 of 10 rows pass the filter, so that each seed has as many groups; the seed shuffles the rows,
    picks the keys of the ranks and the payloads."""
    g = _gen(seed)
    p = 1.0 - W.HC_ZIPF_S
    at = torch.randperm(rows, generator=g, device="cuda")
    pay = _ints(g, 0, 400_000_000, rows)
    for lo in range(0, rows, 1 << 24):  # bounded temporaries
        i = at[lo:lo + (1 << 24)]
        passing = (i * 7919) % 10 < 6
        rank = (1.0 + (i.double() + 0.5) / rows * (float(ranks + 1) ** p - 1.0)).pow_(1.0 / p).long().clamp_(1, ranks)
        at[lo:lo + (1 << 24)] = _mix(rank + 1_000_003 * (int(seed) % 1000))
        pay[lo:lo + (1 << 24)] += torch.where(passing, 0, HC_CUT)
    return at, pay


HC_CUT = 600_000_000


def prepare_hicard(case, seed):
    key, pay = _hicard(case["rows"], case["ranks"], seed)
    cols = [_Raw(abi.T_I64, key), _Raw(abi.T_I64, pay)]
    e = _env(cols)
    aq = q.AggQuery(e, q.col(1).lt(HC_CUT), [(q.col(0), True)],
                    [q.Agg("COUNT"), q.Agg("SUM", q.col(1), "BIGINT", True)])
    return {"cols": cols, "e": e, "aq": aq, "prog": _jit(e, aq.plan, abi.JF_GROUPED),
            "cap": W.plain_capacity(aq.plan, min(case["ranks"], case["rows"])),
            "arrays": estimator.batch_arrays(_batches(cols, case["rows"]))}


def run_hicard(s):
    agg = ops.GpuAggregator(s["aq"].plan, s["cap"])
    _add(agg, s["e"], s["arrays"])
    agg.run(s["e"].env, s["prog"])
    if agg.overflowed():
        raise RuntimeError("hash table overflow")
    kp, ap, g = agg.compact()
    agg.close()
    order = torch.empty(g, dtype=torch.float64, device="cuda")
    ops.bits_to_double(kp, g, order.data_ptr())
    perm = ops.sort_perm([order.data_ptr()], [0], g)
    out = {"key": torch.empty(g, dtype=torch.int64, device="cuda"),
           "count": torch.empty(g, dtype=torch.float64, device="cuda"),
           "sum_low": torch.empty(g, dtype=torch.int64, device="cuda"),
           "sum_high": torch.empty(g, dtype=torch.int64, device="cuda")}
    ops.gather(kp, abi.PT_I64, perm, g, out["key"].data_ptr())
    slots = {"count": 0, "sum_low": s["aq"].aggs[1].slot, "sum_high": s["aq"].aggs[1].hi_slot}
    for name, a in slots.items():
        ops.gather(ap + a * g * 8, abi.PT_I64, perm, g, out[name].data_ptr())
    for p in (kp, ap, perm):
        ops.tmp_free(p)
    return out


def exact_hicard(case, seed):
    key, pay = _hicard(case["rows"], case["ranks"], seed)
    live = pay < HC_CUT
    keys, inv = torch.unique(key[live], return_inverse=True)
    n, pay = keys.numel(), pay[live]
    total = _sum_by(inv, pay, n)
    return {"key": keys, "count": _sum_by(inv, torch.ones_like(pay), n).double(), "sum_low": total & 0xFFFFFFFF,
            "sum_high": total >> 32}


# ---------------------------------------------------------------- selection and gathers
def _select(rows, seed):
    """Prices are a permutation, so that each seed selects as many rows."""
    g = _gen(seed)
    r = torch.randperm(rows, generator=g, device="cuda")
    return (_ints(g, 0, 1 << 40, rows), r.double() * (1000.0 / rows), _ints(g, 5, 2557, rows, torch.int32),
            _ints(g, 0, 200, rows, torch.uint8), r % 20 == 7)


def prepare_select(case, seed):
    ident, price, date, tag, dead = _select(case["rows"], seed)
    cols = [_Raw(abi.T_I64, ident), _Raw(abi.T_F64, price), _Enc(abi.T_I32, 2, date, base=8000),
            _Enc(abi.T_I32, 1, tag, base=-3)]
    e = _env(cols)
    where = e.compile(q.and_(q.col(1).lt(10.0 * case["percent"]), q.col(2).ge(8005)))
    plan = abi.AggPlan()
    plan.hasWhere, plan.where, plan.naggs = 1, where, 1
    plan.ops[0] = abi.AGG_COUNT
    dele = _pack_bits(dead) if case["deleted"] else None
    lens = _segs(case["rows"])
    return {"cols": cols, "dele": dele, "e": e, "where": where, "prog": _jit(e, plan, abi.JF_FLAGM),
            "batches": _batches(cols, case["rows"], dele), "boff": [SEG * s for s in range(len(lens))]}


def run_select(s):
    idx, m, per = ops.select_multi(s["e"].env, s["where"], s["batches"], s["e"].ncols, s["prog"])
    out = {"per_batch": np.array(per, dtype=np.int64), "row": torch.empty(m, dtype=torch.int32, device="cuda")}
    ops.check(ops.lib().ws_d2d(out["row"].data_ptr(), idx, 4 * m))
    for c, (name, ptype, dtype) in enumerate((("ident", abi.PT_I64, torch.int64), ("price", abi.PT_F64, torch.float64),
                                              ("date", abi.PT_I32, torch.int32), ("tag", abi.PT_I32, torch.int32))):
        out[name] = torch.empty(m, dtype=dtype, device="cuda")
        ops.gather_multi([b[2][c] for b in s["batches"]], s["boff"], ptype, out[name].element_size(), idx, m,
                         out[name].data_ptr())
    ops.tmp_free(idx)
    return out


def exact_select(case, seed):
    ident, price, date, tag, dead = _select(case["rows"], seed)
    live = (price < 10.0 * case["percent"]) & (date >= 5)
    if case["deleted"]:
        live &= ~dead
    row = live.nonzero().view(-1)
    per = torch.bincount(row // SEG, minlength=len(_segs(case["rows"])))
    return {"per_batch": per.cpu().numpy(), "row": row.int(), "ident": ident[row], "price": price[row],
            "date": date[row] + 8000, "tag": tag[row].int() - 3}


# ---------------------------------------------------------------- join + aggregate
def _join(case, seed):
    g = _gen(seed)
    nb, npr = case["build"], case["probe"]
    key = torch.randperm(nb, generator=g, device="cuda")
    date = _ints(g, 0, 2406, nb, torch.int32)
    fk = _ints(g, 0, nb, npr)
    if case["sparse"]:
        key, fk = _mix(key + 977), _mix(fk + 977)
    return key, date, fk, _ints(g, 0, 1_000_000, npr), _ints(g, 0, case["groups"], npr, torch.int32)


DATE_CUT = 1203  # half of the build rows pass


def prepare_join(case, seed):
    key, date, fk, cents, gkey = _join(case, seed)
    build = [_Raw(abi.T_I64, key), _Raw(abi.T_I32, date)]
    eb = _env(build)
    where = eb.compile(q.col(1).lt(DATE_CUT))
    fp = abi.AggPlan()
    fp.hasWhere, fp.where, fp.naggs = 1, where, 1
    fp.ops[0] = abi.AGG_COUNT
    ej = q.Env()
    aggs = [q.Agg("COUNT"), q.Agg("SUM", q.col(1), "BIGINT", True)]
    ej.column(abi.T_I32)
    ej.column(abi.T_I64)
    if case["left"]:
        ej.column(abi.T_I32N)
        aggs += [q.Agg("COUNT", q.col(2), "INT", True, nullable=True), q.Agg("MAX", q.col(2), "INT", True, nullable=True)]
    aq = q.AggQuery(ej, None, [(q.col(0), True)], aggs)
    ds = q.dense_spec(aq.plan, [(0, case["groups"] - 1)], case["probe"])
    return {"build": build, "fk": fk, "cents": cents, "gkey": gkey, "eb": eb, "where": where, "ej": ej, "aq": aq,
            "ds": ds, "left": case["left"], "cap": W.plain_capacity(aq.plan, case["groups"]),
            "batches": _batches(build, case["build"]), "fprog": _jit(eb, fp, abi.JF_FLAGM),
            "aprog": _jit(ej, aq.plan, abi.JF_GROUPED if ds is None else abi.JF_DENSE)}


def run_join(s):
    key, date = s["build"]
    idx, mb, _ = ops.select_multi(s["eb"].env, s["where"], s["batches"], s["eb"].ncols, s["fprog"])
    bkey = torch.empty(mb, dtype=torch.int64, device="cuda")
    ops.gather(key.x.data_ptr(), abi.PT_I64, idx, mb, bkey.data_ptr())
    bview = abi.ColView(bkey.data_ptr(), abi.T_I64, 0, 0, 0)
    pview = abi.ColView(s["fk"].data_ptr(), abi.T_I64, 0, 0, 0)
    join = ops.hash_join_outer if s["left"] else ops.hash_join
    ob, op, m = join(bview, mb, pview, s["fk"].numel())
    gkey = torch.empty(m, dtype=torch.int32, device="cuda")
    cents = torch.empty(m, dtype=torch.int64, device="cuda")
    ops.gather(s["gkey"].data_ptr(), abi.PT_I32, op, m, gkey.data_ptr())
    ops.gather(s["cents"].data_ptr(), abi.PT_I64, op, m, cents.data_ptr())
    views = [abi.ColView(gkey.data_ptr(), abi.T_I32, 0, 0, 0), abi.ColView(cents.data_ptr(), abi.T_I64, 0, 0, 0)]
    if s["left"]:
        bdate = torch.empty(mb, dtype=torch.int32, device="cuda")
        ops.gather(date.x.data_ptr(), abi.PT_I32, idx, mb, bdate.data_ptr())
        jdate = torch.empty(m, dtype=torch.int32, device="cuda")
        ops.gather_null(bdate.data_ptr(), abi.PT_I32, ob, m, jdate.data_ptr())
        views.append(abi.ColView(jdate.data_ptr(), abi.T_I32N, 0, 0, 0))
    agg = ops.GpuAggregator(s["aq"].plan, s["cap"], s["ds"])
    agg.add_batches(s["ej"].ncols, [(m, 0, views)])
    agg.run(s["ej"].env, s["aprog"])
    if agg.overflowed():
        raise RuntimeError("hash table overflow")
    keys, accs, _ = agg.fetch(exact=False)
    agg.close()
    for p in (idx, ob, op):
        ops.tmp_free(p)
    if s["ds"] is None:
        order = np.lexsort(keys.view(np.int64).T)
        keys, accs = keys[order], accs[order]
    # the groups as the engine takes them: every slot's 64 bits (counts and INT maxima are doubles, a BIGINT SUM
    # its low 32 bits and the rest)
    return {"keys": keys.view(np.int64), "slots": accs.view(np.int64)}


def exact_join(case, seed):
    key, date, fk, cents, gkey = _join(case, seed)
    if case["sparse"]:
        order = torch.argsort(key)
        at = order[torch.searchsorted(key[order], fk)]
    else:
        inverse = torch.empty_like(key)
        inverse[key] = torch.arange(key.numel(), device="cuda")
        at = inverse[fk]
    d = date[at].long()
    hit = d < DATE_CUT
    use = torch.ones_like(hit) if case["left"] else hit
    keys, inv = torch.unique(gkey[use].long(), return_inverse=True)
    n = keys.numel()
    total = _sum_by(inv, cents[use], n)
    count = _sum_by(inv, torch.ones_like(inv), n).double()
    slots = [count.view(torch.int64), total & 0xFFFFFFFF, total >> 32]
    if case["left"]:
        none = torch.iinfo(torch.int64).min
        top = _min_by(inv, torch.where(hit, d, none), n, "amax")
        slots += [_sum_by(inv, hit.long(), n).double().view(torch.int64),
                  torch.where(top == none, float("-inf"), top.double()).view(torch.int64)]
    return {"keys": keys.view(-1, 1).cpu().numpy(), "slots": torch.stack(slots, 1).cpu().numpy()}


# ---------------------------------------------------------------- ORDER BY
def _orderby(rows, seed):
    g = _gen(seed)
    return _ints(g, 900, 105_001, rows) * 100, _ints(g, 0, 11, rows), _ints(g, 8000, 10557, rows, torch.int32)


def prepare_orderby(case, seed):
    price, disc, date = _orderby(case["rows"], seed)
    cols = [_Raw(abi.T_I64, price), _Raw(abi.T_I64, disc), _Raw(abi.T_I32, date)]
    e = _env(cols)
    p1 = e.compile(q.col(0) * (q.ilit(100) - q.col(1)) / q.lit(100.0))
    p2 = e.compile(q.col(2))
    for slot, c in enumerate(cols):
        e.bind(slot, c.x.data_ptr())
    return {"cols": cols, "e": e, "p1": p1, "p2": p2}


def run_orderby(s):
    e, n = s["e"], s["cols"][0].x.numel()
    k1 = torch.empty(n, dtype=torch.float64, device="cuda")
    k2 = torch.empty(n, dtype=torch.float64, device="cuda")
    ops.eval_at(e.env, e.ncols, s["p1"], None, n, k1.data_ptr())
    ops.eval_at(e.env, e.ncols, s["p2"], None, n, k2.data_ptr())
    perm = ops.sort_perm([k1.data_ptr(), k2.data_ptr()], [1, 0], n)
    out = {"row": torch.empty(n, dtype=torch.int32, device="cuda"),
           "revenue": torch.empty(n, dtype=torch.float64, device="cuda"),
           "date": torch.empty(n, dtype=torch.int32, device="cuda")}
    ops.check(ops.lib().ws_d2d(out["row"].data_ptr(), perm, 4 * n))
    ops.gather(k1.data_ptr(), abi.PT_F64, perm, n, out["revenue"].data_ptr())
    ops.gather(s["cols"][2].x.data_ptr(), abi.PT_I32, perm, n, out["date"].data_ptr())
    ops.tmp_free(perm)
    return out


def exact_orderby(case, seed):
    price, disc, date = _orderby(case["rows"], seed)
    rev = (price * (100 - disc)).double() / 100.0
    row = torch.argsort(date, stable=True)
    row = row[torch.argsort(rev[row], descending=True, stable=True)]
    return {"row": row.int(), "revenue": rev[row], "date": date[row]}


# ---------------------------------------------------------------- segment encoding
def prepare_encode(case, seed):
    n, g = case["rows"], _gen(seed)
    date = _ints(g, 8000, 10557, n, torch.int32)
    cents = _ints(g, 90_000, 10_500_001, n)
    price = cents.double() / 100.0                                    # decimal doubles
    disc = torch.tensor(DISCOUNTS, dtype=torch.float64, device="cuda")[_ints(g, 0, 11, n)]  # few distinct values
    batch = torch.sort(_ints(g, 0, max(1, n // 500), n))[0]           # long runs
    return {"engine": [(date, abi.PT_I32), (cents, abi.PT_I64), (price, abi.PT_F64), (disc, abi.PT_F64)],
            "own": [(date, abi.T_I32), (batch, abi.T_I64)]}


def run_encode(s):
    def keep(ptr, nbytes):
        out = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        ops.check(ops.lib().ws_d2d(out.data_ptr(), ptr, nbytes))
        ops.tmp_free(ptr)
        return out
    out = {}
    for i, (x, ptype) in enumerate(s["engine"]):
        ptr, nbytes, enc = ops.encode_column_engine(x.data_ptr(), ptype, x.numel())
        out["engine%d" % i], out["engine%d_enc" % i] = keep(ptr, nbytes), enc
    for i, (x, t) in enumerate(s["own"]):
        ptr, nbytes, enc = ops.encode_column(x.data_ptr(), t, x.numel())
        out["own%d" % i], out["own%d_enc" % i] = keep(ptr, nbytes), enc
    return out


# ---------------------------------------------------------------- the interface
def prepare(case, seed):
    return {"kind": case["kind"], "state": globals()["prepare_" + case["kind"]](case, int(seed))}


def run(state):
    return globals()["run_" + state["kind"]](state["state"])


def exact(case, seed):
    if case["kind"] == "encode":
        return None  # bytes, compared as they are
    return globals()["exact_" + case["kind"]](case, int(seed))


def work(case):
    kind = case["kind"]
    group_bytes = {"prepared": 7 * 8, "burst": 7 * 8, "query": 7 * 8, "dense": 8 * 8}  # key + aggregates
    if kind == "burst":
        return {"bytes": sum(_burst_sizes(case)) * 20 + case["queries"] * case["groups"] * group_bytes[kind], "flops": 0}
    if kind in ("prepared", "query"):
        return {"bytes": case["rows"] * (20 if case.get("keys", 1) == 1 else 24) + case["groups"] * group_bytes[kind],
                "flops": 0}
    if kind == "pricing":
        return {"bytes": case["rows"] * W.PRICING_BYTES_PER_ROW + 6 * 12 * 8, "flops": 0}
    if kind == "scan":
        return {"bytes": int(case["rows"] * (2 + 1 + 8 + 1 + 2 + (0.125 if case["deleted"] else 0))), "flops": 0}
    if kind == "dense":
        return {"bytes": case["rows"] * 24 + case["groups"] * group_bytes[kind], "flops": 0}
    if kind == "hicard":
        return {"bytes": case["rows"] * W.HC_BYTES_PER_ROW + int(0.4 * min(case["ranks"], case["rows"])) * 32, "flops": 0}
    if kind == "select":
        m = int(case["rows"] * case["percent"] / 100)
        return {"bytes": case["rows"] * 10 + m * (4 + 8 + 8 + 4 + 4 + 8 + 1), "flops": 0}
    if kind == "join":
        nb, npr = case["build"], case["probe"]
        m = npr if case["left"] else npr // 2
        return {"bytes": nb * 8 + npr * 8 + m * 12 + case["groups"] * 32, "flops": 0}
    if kind == "orderby":
        return {"bytes": case["rows"] * (8 + 8 + 4 + 4 + 8 + 4), "flops": 0}
    return {"bytes": case["rows"] * (4 + 8 + 8 + 8 + 4 + 8 + 2 + 4 + 4 + 1 + 2), "flops": 0}
