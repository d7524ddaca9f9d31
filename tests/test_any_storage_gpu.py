"""Batches stored otherwise than their plan's hints, plans compiled in the background (the default mode): runs, a
multi-query launch and a prepared query give the oracle's groups, and a process may end as soon as its plan was used."""
import os
import subprocess
import sys
import time

import numpy as np
import pytest

from oracle import oracle
from warpstore_b200 import abi, estimator, ops
from warpstore_b200 import query as q
from warpstore_b200 import workloads as W

from .helpers import compare_exact

pytestmark = pytest.mark.gpu


def prepared(kind, stored, seed):
    """A plan of columns hinted as encoding 2, and batches of which the second is stored as `stored`."""
    rng = np.random.default_rng(seed)
    e = q.Env()
    e.column(abi.T_I32, 0, 0)
    e.column(abi.T_I64, 0, 2)
    aggs = [q.Agg("COUNT"), q.Agg("SUM", q.col(1), "BIGINT", True), q.Agg("MAX", q.col(1), "BIGINT", True),
            q.Agg("MIN", q.col(1), "BIGINT", True)]
    aq = q.AggQuery(e, q.col(1).lt(30_000), [(q.col(0), True)], aggs)
    ds = None
    if kind == "dense":
        ds = abi.DenseSpec()
        ds.G, ds.kmin[0], ds.range[0], ds.stride[0] = 9, 0, 9, 1
    host, dev, keep = [], [], []
    for b, n in enumerate((5000, 1027, 3001)):
        k, v = rng.integers(0, 9, n).astype(np.int32), rng.integers(0, 60_000, n)
        enc = stored if b == 1 else 2
        raw = W.encode_for(v, enc)[0] if enc else v.view(np.uint8)
        db = [ops.DeviceBuffer.from_array(k), ops.DeviceBuffer.from_array(raw)]
        keep += [k, raw, db]
        host.append((n, 0, [abi.ColView(k.ctypes.data, abi.T_I32, 0, 0, 0), abi.ColView(raw.ctypes.data, abi.T_I64, 0, enc, 0)]))
        dev.append((n, 0, [abi.ColView(db[0].ptr, abi.T_I32, 0, 0, 0), abi.ColView(db[1].ptr, abi.T_I64, 0, enc, 0)]))
    return e, aq, ds, host, dev, keep


@pytest.mark.parametrize("kind", ["hash", "dense"])
def test_runs_of_background_plans(kind):
    e, aq, ds, host, dev, keep = prepared(kind, 0, 1)
    fn = abi.JF_DENSE if kind == "dense" else abi.JF_GROUPED
    ok, ow, _ = oracle.aggregate(e.env, aq.plan, host, e.ncols)
    ops.jit_set_mode(abi.JIT_ON)
    try:
        prog, t0 = None, time.time()
        while not prog and time.time() - t0 < 120:
            prog = ops.jit_get(e.env, e.ncols, aq.plan, fn, "test")
            time.sleep(0.01)
        assert prog
        t0 = time.time()
        while time.time() - t0 < 1:
            agg = ops.GpuAggregator(aq.plan, 64, ds)
            agg.add_batches(e.ncols, dev)
            agg.run(e.env, prog)
            k, _, x = agg.fetch()
            compare_exact(aq.plan, k, x, ok, ow)
            agg.close()
            time.sleep(0.1)
        aggs = [ops.GpuAggregator(aq.plan, 64, ds) for _ in range(2)]
        for a in aggs:
            a.add_batches(e.ncols, dev)
        ops.agg_run_many(aggs, [e.env, e.env], prog)
        for a in aggs:
            k, _, x = a.fetch()
            compare_exact(aq.plan, k, x, ok, ow)
            a.close()
        ex = ops.Executor(aq.plan, 64, ds, e.env, e.ncols, estimator.batch_arrays(dev), prog, 64)
        ex.run(e.env)
        ops.sync()
        k, x, st = ex.results()
        assert not st["overflow"] and not st["error"]
        compare_exact(aq.plan, k, x, ok, ow)
        ex.close()
    finally:
        ops.jit_set_mode(-1)


def test_a_prepared_query_of_a_new_plan():
    e, aq, ds, host, dev, keep = prepared("hash", 0, 2)
    aq = q.AggQuery(e, q.col(1).lt(200), [(q.col(0), True)], [q.Agg("COUNT"), q.Agg("MIN", q.col(1), "BIGINT", True)])
    raw = [np.random.default_rng(9).integers(0, 250, n) for n in (4000, 77)]
    host, dev = [], []
    for n, v, enc in zip((4000, 77), raw, (2, 1)):
        k = (v % 9).astype(np.int32)
        seg = W.encode_for(v, enc)[0]
        db = [ops.DeviceBuffer.from_array(k), ops.DeviceBuffer.from_array(seg)]
        keep += [k, seg, db]
        host.append((n, 0, [abi.ColView(k.ctypes.data, abi.T_I32, 0, 0, 0), abi.ColView(seg.ctypes.data, abi.T_I64, 0, enc, 0)]))
        dev.append((n, 0, [abi.ColView(db[0].ptr, abi.T_I32, 0, 0, 0), abi.ColView(db[1].ptr, abi.T_I64, 0, enc, 0)]))
    ok, ow, _ = oracle.aggregate(e.env, aq.plan, host, e.ncols)
    ops.jit_set_mode(abi.JIT_ON)
    try:
        prog, t0 = None, time.time()
        while not prog and time.time() - t0 < 120:
            prog = ops.jit_get(e.env, e.ncols, aq.plan, abi.JF_GROUPED, "test")
        assert prog
        ex = ops.Executor(aq.plan, 64, None, e.env, e.ncols, estimator.batch_arrays(dev), prog, 64)
        ex.run(e.env)
        ops.sync()
        k, x, _ = ex.results()
        compare_exact(aq.plan, k, x, ok, ow)
        ex.close()
    finally:
        ops.jit_set_mode(-1)


CHILD = r"""
import time
import numpy as np
from warpstore_b200 import abi, ops
from warpstore_b200 import query as q
e = q.Env()
e.column(abi.T_I32, 0, 0)
e.column(abi.T_I64, 0, 2)
aq = q.AggQuery(e, q.col(1).lt(300), [(q.col(0), True)], [q.Agg("COUNT"), q.Agg("SUM", q.col(1), "BIGINT", True)])
prog = None
while not prog:
    prog = ops.jit_get(e.env, e.ncols, aq.plan, abi.JF_GROUPED, "test")
    time.sleep(0.005)
k, v = np.arange(5000, dtype=np.int32) % 7, np.arange(5000) % 500
bufs = [ops.DeviceBuffer.from_array(x) for x in (k, v)]
agg = ops.GpuAggregator(aq.plan, 64)
agg.add_batches(e.ncols, [(5000, 0, [abi.ColView(bufs[0].ptr, abi.T_I32, 0, 0, 0), abi.ColView(bufs[1].ptr, abi.T_I64, 0, 0, 0)])])
agg.run(e.env, prog)
assert agg.fetch()[0].shape == (7, 1)
agg.close()
"""


def test_a_process_may_end_after_its_first_run():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    for _ in range(2):
        r = subprocess.run([sys.executable, "-c", CHILD], cwd=root, env=dict(os.environ, PYTHONPATH=root), capture_output=True,
                           text=True, timeout=120)
        assert r.returncode == 0, r.stderr[-2000:]
