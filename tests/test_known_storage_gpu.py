"""Compiled scans of columns with known storage: the packed fetch, the narrow integer evaluation and the
compact shared tables where they can go wrong — values around 2^31 and 2^62, constants that do not fit in
int32, NULLs, segments stored otherwise than hinted, unaligned views, ragged batches, every scan kind, few and
many groups — against the CPU oracle; and the one-pass selection with its gathers against numpy."""
import numpy as np
import pytest

from oracle import oracle
from warpstore_b200 import abi, ops
from warpstore_b200 import query as q
from warpstore_b200 import workloads as W

from .helpers import compare_exact

pytestmark = pytest.mark.gpu


def columns(n, values, rng):
    if values == "small":
        v, w = rng.integers(-1000, 1000, n), rng.integers(0, 100, n)
    elif values == "edge32":
        v = rng.choice([-2**31, 2**31 - 1, -2**31 - 1, 2**31, 0, -1, 46341, 10**9], n)
        w = rng.integers(-2, 3, n)
    else:  # "wide": sums leave int64, products do not
        v, w = rng.choice([2**61, -2**61, 2**62 - 1, 5, -7], n), rng.integers(-1, 2, n)
    return v.astype(np.int64), w.astype(np.int64)


def program(e, plan, fn):
    ops.jit_set_mode(abi.JIT_SYNC)
    try:
        prog = ops.jit_get(e.env, e.ncols, plan, fn, "test")
    finally:
        ops.jit_set_mode(-1)
    assert prog, "codegen failed"
    return prog


@pytest.mark.parametrize("values,const", [("small", 100), ("edge32", 3), ("edge32", 2**31 + 7), ("wide", 0)])
@pytest.mark.parametrize("kind,groups", [("nokeys", 1), ("dense", 3), ("dense", 40), ("dense", 3000), ("dense", 60_000),
                                         ("hash", 3), ("hash", 500), ("hash", 5000)])
def test_narrow_and_wide_values(values, const, kind, groups):
    rng = np.random.default_rng(groups + const % 1000)
    sizes = [30_011, 1, 1023, 1025, 5]
    n = sum(sizes)
    v, w = columns(n, values, rng)
    k = rng.integers(-5, groups - 5, n).astype(np.int32)
    f = rng.standard_normal(n)
    d = rng.integers(0, 250, n)
    nul = np.where(rng.random(n) < 0.2, abi.NULL_I64, v % 1000)
    for hinted, stored in ((1, 1), (1, 2)):  # segments as hinted, and one stored in another width
        e = q.Env()
        for t, enc in ((abi.T_I32, 0), (abi.T_I64, 0), (abi.T_I64, 0), (abi.T_F64, 0), (abi.T_I64, hinted), (abi.T_I64N, 0)):
            e.column(t, 0, enc)
        ovf = ops.DeviceBuffer.from_array(np.zeros(1, np.int32))  # the engine's overflow flag: no product below overflows
        e.env.ovf = ovf.ptr
        prod = q.col(1) * (q.ilit(const) - q.col(2)) if values != "wide" else q.col(1) * q.col(2)
        aggs = [q.Agg("COUNT"), q.Agg("SUM", q.col(1), "BIGINT", True), q.Agg("SUM", prod, "BIGINT", False),
                q.Agg("MIN", prod, "BIGINT", False), q.Agg("MAX", q.col(4), "BIGINT", True),
                q.Agg("MAX", q.col(3), "DOUBLE", True), q.Agg("SUM", q.col(5), "BIGINT", True, nullable=True)]
        keys = [] if kind == "nokeys" else [(q.col(0), True)]
        aq = q.AggQuery(e, q.col(4).lt(200), keys, aggs)
        ds = None
        if kind == "dense":
            ds = abi.DenseSpec()
            ds.G, ds.kmin[0], ds.range[0], ds.stride[0] = groups, -5, groups, 1
        prog = program(e, aq.plan, {"nokeys": abi.JF_NOKEYS, "dense": abi.JF_DENSE, "hash": abi.JF_GROUPED}[kind])
        host, dev, keep, at = [], [], [], 0
        for b, m in enumerate(sizes):
            enc = stored if b == 1 else hinted
            pad = 8 if b == 2 else 0  # an unaligned batch: views that no 16-byte load may touch
            hv, dv = [], []
            for x, t, en in ((k, abi.T_I32, 0), (v, abi.T_I64, 0), (w, abi.T_I64, 0), (f, abi.T_F64, 0), (d, abi.T_I64, enc),
                             (nul, abi.T_I64N, 0)):
                part = np.ascontiguousarray(x[at:at + m])
                raw = W.encode_for(part, en)[0] if en else part.view(np.uint8)
                buf = np.zeros(raw.size + 64, np.uint8)
                buf[pad if not en else 0:][:raw.size] = raw
                db = ops.DeviceBuffer.from_array(buf)
                keep += [buf, db]
                off = pad if not en else 0
                hv.append(abi.ColView(buf.ctypes.data + off, t, 0, en, 0))
                dv.append(abi.ColView(db.ptr + off, t, 0, en, 0))
            host.append((m, 0, hv))
            dev.append((m, 0, dv))
            at += m
        ok, ow, _ = oracle.aggregate(e.env, aq.plan, host, e.ncols)
        agg = ops.GpuAggregator(aq.plan, 1 << max(10, (2 * groups - 1).bit_length()), ds)
        agg.add_batches(e.ncols, dev)
        agg.run(e.env, prog)
        assert not agg.overflowed()
        gk, _, gx = agg.fetch()
        compare_exact(aq.plan, gk, gx, ok, ow)
        assert ovf.to_array(np.int32)[0] == 0
        agg.close()


@pytest.mark.parametrize("sizes", [[1], [31, 1, 1024], [4096, 1023, 7, 100_003], [1025] * 5])
@pytest.mark.parametrize("percent", [0, 3, 60, 100])
def test_selection_and_gathers(sizes, percent):
    rng = np.random.default_rng(sum(sizes) + percent)
    n = sum(sizes)
    a = rng.integers(0, 100, n)
    code = rng.integers(0, 60_000, n)
    dbl = rng.choice(np.array([0.25, 1.5, -3.0]), n)
    gone = rng.random(n) < 0.1
    e = q.Env()
    for t, enc in ((abi.T_I64, 0), (abi.T_I32, 2), (abi.T_F64, 0)):
        e.column(t, 0, enc)
    where = e.compile(q.and_(q.col(0).lt(percent), q.col(1).ge(-7)))
    plan = abi.AggPlan()
    plan.hasWhere, plan.where, plan.naggs = 1, where, 1
    plan.ops[0] = abi.AGG_COUNT
    prog = program(e, plan, abi.JF_FLAGM)
    batches, keep, at, boff = [], [], 0, []
    for m in sizes:
        bits = np.zeros((m + 31) // 32 * 32, np.uint8)
        bits[:m] = gone[at:at + m]
        bufs = [ops.DeviceBuffer.from_array(x) for x in
                (a[at:at + m], W.encode_for(code[at:at + m] - 7, 2)[0], dbl[at:at + m],
                 np.packbits(bits, bitorder="little").view(np.uint32))]
        keep += bufs
        views = [abi.ColView(bufs[0].ptr, abi.T_I64, 0, 0, 0), abi.ColView(bufs[1].ptr, abi.T_I32, 0, 2, 0),
                 abi.ColView(bufs[2].ptr, abi.T_F64, 0, 0, 0)]
        batches.append((m, bufs[3].ptr, views))
        boff.append(at)
        at += m
    idx, m, per = ops.select_multi(e.env, where, batches, e.ncols, prog)
    want = np.flatnonzero((a < percent) & ~gone)
    got = ops.device_to_array(idx, np.int32, m)
    assert np.array_equal(got, want)
    assert per == [int(((want >= o) & (want < o + s)).sum()) for o, s in zip(boff, sizes)]
    ops.tmp_free(idx)
    for order in (want, want[::-1], rng.integers(0, n, 1003)):  # ascending, descending, any
        for skip in (0, 1):  # an index array off the 16-byte boundary
            di = ops.DeviceBuffer.from_array(np.concatenate([np.zeros(skip, np.int32), order.astype(np.int32)]))
            for c, (pt, src) in enumerate(((abi.PT_I64, a), (abi.PT_I32, code - 7), (abi.PT_F64, dbl))):
                dt = {abi.PT_I64: np.int64, abi.PT_I32: np.int32, abi.PT_F64: np.float64}[pt]
                out = ops.DeviceBuffer(order.size * np.dtype(dt).itemsize + 16)
                ops.gather_multi([b[2][c] for b in batches], boff, pt, np.dtype(dt).itemsize, di.ptr + 4 * skip, order.size,
                                 out.ptr)
                assert np.array_equal(out.to_array(dt, order.size), src[order].astype(dt))
