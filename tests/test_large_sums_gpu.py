"""Integer SUMs of large arguments (microsecond timestamps, scaled products) in the shared-memory GROUP BY tables:
exact past int64 in both directions, and aggregated on chip like small ones."""
import time

import numpy as np
import pytest

from oracle import oracle
from warpstore_b200 import abi, ops
from warpstore_b200 import query as q

from .helpers import compare_exact

pytestmark = pytest.mark.gpu


def query(kind, groups):
    e = q.Env()
    for t in (abi.T_I32, abi.T_I64, abi.T_I64N):
        e.column(t, 0, 0)
    aggs = [q.Agg("COUNT"), q.Agg("SUM", q.col(1), "BIGINT", True), q.Agg("MIN", q.col(1), "BIGINT", True),
            q.Agg("SUM", q.col(2), "BIGINT", True, nullable=True)]
    aq = q.AggQuery(e, None, [(q.col(0), True)], aggs)
    ds = None
    if kind == "dense":
        ds = abi.DenseSpec()
        ds.G, ds.kmin[0], ds.range[0], ds.stride[0] = groups, 0, groups, 1
    ops.jit_set_mode(abi.JIT_SYNC)
    try:
        prog = ops.jit_get(e.env, e.ncols, aq.plan, abi.JF_DENSE if kind == "dense" else abi.JF_GROUPED, "test")
    finally:
        ops.jit_set_mode(-1)
    assert prog, "codegen failed"
    return e, aq, ds, prog


def columns(n, groups, values, rng):
    v = {"small": lambda: rng.integers(0, 1000, n), "negative": lambda: rng.integers(-1000, 0, n),
         "mixed": lambda: rng.integers(-2**33, 2**33, n), "stamps": lambda: rng.integers(2**50, 2**51, n),
         "limits": lambda: rng.choice(np.array([2**63 - 1, -2**63 + 1, -1, 0, 1, 2**32, -2**32, 2**62], np.int64), n),
         "top": lambda: np.full(n, 2**63 - 1), "bottom": lambda: np.full(n, -2**63 + 1)}[values]().astype(np.int64)
    nul = np.where(rng.random(n) < 0.3, abi.NULL_I64, v)
    return rng.integers(0, groups, n).astype(np.int32), v, nul


def aggregate(e, aq, ds, prog, cap, bufs, n):
    agg = ops.GpuAggregator(aq.plan, cap, ds)
    agg.add_batches(e.ncols, [(n, 0, [abi.ColView(b.ptr, t, 0, 0, 0) for b, t in
                                      zip(bufs, (abi.T_I32, abi.T_I64, abi.T_I64N))])])
    agg.run(e.env, prog)
    return agg


@pytest.mark.parametrize("values", ["small", "negative", "mixed", "stamps", "limits", "top", "bottom"])
@pytest.mark.parametrize("kind,groups", [("hash", 3), ("hash", 400), ("dense", 30), ("dense", 2000)])
def test_exact(kind, groups, values):
    n = 300_007
    e, aq, ds, prog = query(kind, groups)
    cols = columns(n, groups, values, np.random.default_rng(groups))
    host = [(n, 0, [abi.ColView(c.ctypes.data, t, 0, 0, 0) for c, t in zip(cols, (abi.T_I32, abi.T_I64, abi.T_I64N))])]
    ok, ow, _ = oracle.aggregate(e.env, aq.plan, host, e.ncols)
    agg = aggregate(e, aq, ds, prog, 1024, [ops.DeviceBuffer.from_array(c) for c in cols], n)
    assert not agg.overflowed()
    keys, _, exact = agg.fetch()
    compare_exact(aq.plan, keys, exact, ok, ow)
    agg.close()


@pytest.mark.parametrize("kind,groups", [("hash", 16), ("dense", 40)])
def test_large_arguments_stay_on_chip(kind, groups):
    """Rows of large arguments cost about what rows of small ones do (a row sent to the global table or its L2
    atomics costs 30 to 50 times as much when few groups take them all)."""
    n = 8_000_000
    e, aq, ds, prog = query(kind, groups)
    best = {}
    for values in ("small", "stamps"):
        bufs = [ops.DeviceBuffer.from_array(c) for c in columns(n, groups, values, np.random.default_rng(1))]
        for rep in range(6):
            agg = ops.GpuAggregator(aq.plan, 1024, ds)
            agg.add_batches(e.ncols, [(n, 0, [abi.ColView(b.ptr, t, 0, 0, 0) for b, t in
                                              zip(bufs, (abi.T_I32, abi.T_I64, abi.T_I64N))])])
            ops.sync()
            t0 = time.perf_counter()
            agg.run(e.env, prog)
            ops.sync()
            dt = time.perf_counter() - t0
            agg.close()
            best[values] = min(best.get(values, 1e9), dt) if rep else 1e9
    assert best["stamps"] < 4 * best["small"], best
