"""Hash GROUP BY of wide plans (compiled and interpreted, one and two keys) and of under-sized tables: against the CPU
oracle, and within a bound of what narrow plans and large tables cost."""
import time

import numpy as np
import pytest

from oracle import oracle
from warpstore_b200 import abi, ops
from warpstore_b200 import query as q

from .helpers import compare_exact

pytestmark = pytest.mark.gpu
WIDE = 24  # argument columns: views of two buffers, each a row further on


def query(aggregates, keys):
    e = q.Env()
    for t in [abi.T_I32, abi.T_I32, abi.T_F64] + [abi.T_I64, abi.T_I64N] * (WIDE // 2):
        e.column(t, 0, 0)
    aggs = [q.Agg("COUNT")]
    for i in range(aggregates):
        c = 3 + i % WIDE
        aggs.append(q.Agg("SUM" if i < WIDE and i % 6 != 5 else "MIN", q.col(c), "BIGINT", True, nullable=c % 2 == 0))
    return e, q.AggQuery(e, q.col(2).lt(0.9), [(q.col(k), True) for k in range(keys)], aggs)


def program(e, aq, jit):
    if not jit:
        return None
    ops.jit_set_mode(abi.JIT_SYNC)
    try:
        prog = ops.jit_get(e.env, e.ncols, aq.plan, abi.JF_GROUPED, "test")
    finally:
        ops.jit_set_mode(-1)
    assert prog, "codegen failed"
    return prog


def columns(n, groups, keys, seed=0):
    rng = np.random.default_rng(seed)
    per = max(1, round(groups ** (1 / keys)))
    v = rng.integers(-2**40, 2**40, n + WIDE)
    return [rng.integers(0, per, n).astype(np.int32), rng.integers(0, per, n).astype(np.int32), rng.random(n), v,
            np.where(rng.random(n + WIDE) < 0.2, abi.NULL_I64, v)]


def batches(bufs, n):
    ptr = [b.ptr if isinstance(b, ops.DeviceBuffer) else b.ctypes.data for b in bufs]
    cols = [(ptr[0], abi.T_I32, 4), (ptr[1], abi.T_I32, 4), (ptr[2], abi.T_F64, 8)]
    for i in range(WIDE):
        cols.append((ptr[3 + i % 2] + 8 * i, abi.T_I64N if i % 2 else abi.T_I64, 8))
    return [(min(70_001, n - at), 0, [abi.ColView(p + at * w, t, 0, 0, 0) for p, t, w in cols])
            for at in range(0, n, 70_001)]


@pytest.mark.parametrize("jit,aggregates", [(True, 4), (True, 10), (True, 16), (True, 26), (False, 3), (False, 6)])
@pytest.mark.parametrize("keys,groups", [(1, 9), (1, 900), (1, 40_000), (2, 36), (2, 2_500)])
def test_wide_plans(jit, aggregates, keys, groups):
    n = 250_013
    e, aq = query(aggregates, keys)
    cols = columns(n, groups, keys)
    ok, ow, _ = oracle.aggregate(e.env, aq.plan, batches(cols, n), e.ncols)
    bufs = [ops.DeviceBuffer.from_array(c) for c in cols]
    agg = ops.GpuAggregator(aq.plan, 1 << max(10, (2 * groups - 1).bit_length()))
    agg.add_batches(e.ncols, batches(bufs, n))
    agg.run(e.env, program(e, aq, jit))
    assert not agg.overflowed()
    k, _, x = agg.fetch()
    compare_exact(aq.plan, k, x, ok, ow)
    agg.close()


def seconds(e, aq, prog, cap, bufs, n):
    best = 1e9
    for _ in range(5):
        agg = ops.GpuAggregator(aq.plan, cap)
        agg.add_batches(e.ncols, batches(bufs, n))
        ops.sync()
        t0 = time.perf_counter()
        agg.run(e.env, prog)
        ops.sync()
        best = min(best, time.perf_counter() - t0)
        over = agg.overflowed()
        agg.close()
    return best, over


@pytest.mark.parametrize("jit,narrow,wide", [(True, 8, 22), (False, 2, 6)])
def test_wide_plans_aggregate_on_chip(jit, narrow, wide):
    """Few groups: without a shared-memory table a plan of twice the aggregates takes 20 times as long."""
    n = 4_000_000
    bufs = [ops.DeviceBuffer.from_array(c) for c in columns(n, 16, 2)]
    t = {}
    for aggregates in (narrow, wide):
        e, aq = query(aggregates, 2)
        t[aggregates] = seconds(e, aq, program(e, aq, jit), 1024, bufs, n)[0]
    assert t[wide] < 6 * t[narrow], t


@pytest.mark.parametrize("jit", [True, False])
def test_a_small_table_overflows_early(jit):
    """A run into a table too small for its groups ends soon after the table is 70 % full (the caller reruns with a larger
    one): it takes no longer than the run with the larger table."""
    n = 6_000_000
    rng = np.random.default_rng(3)
    cols = columns(n, 4, 1)
    cols[0] = rng.integers(0, 2_000_000, n).astype(np.int32)
    bufs = [ops.DeviceBuffer.from_array(c) for c in cols]
    e, aq = query(2, 1)
    prog = program(e, aq, jit)
    small, over = seconds(e, aq, prog, 1 << 17, bufs, n)
    assert over
    large, over = seconds(e, aq, prog, 1 << 22, bufs, n)
    assert not over
    assert small < 2 * large, (small, large)
