"""Result delivery where its paths change and at their edges: the one-launch form (at most 4097 result rows)
and the counted form, chunk boundaries, ranges of fetch_async, the key that equals the hash table's empty
marker, groups at both ends of a dense range — fetch, fetch_async and compact against numpy."""
import numpy as np
import pytest

from warpstore_b200 import abi, ops
from warpstore_b200 import query as q

pytestmark = pytest.mark.gpu


def expected(k, v, f):
    keys, inv = np.unique(k, return_inverse=True)
    s = np.zeros(keys.size, np.int64)
    np.add.at(s, inv, v)
    m = np.full(keys.size, np.iinfo(np.int64).max)
    np.minimum.at(m, inv, v)
    fm = np.full(keys.size, -np.inf)
    np.maximum.at(fm, inv, f)
    return keys, np.bincount(inv).astype(np.int64), s, m, fm


@pytest.mark.parametrize("dense,size,present", [
    (True, 1, "all"), (True, 4096, "ends"), (True, 4097, "all"), (True, 4098, "ends"), (True, 6144, "some"),
    (True, 70_001, "some"), (True, 4098, "none"),
    (False, 1024, "all"), (False, 4096, "some"), (False, 8192, "some"), (False, 1 << 17, "all")])
def test_delivery(dense, size, present):
    rng = np.random.default_rng(size)
    n = 60_000
    if dense:
        pool = {"all": np.arange(size), "ends": np.array([0, size - 1]), "none": np.arange(1),
                "some": np.unique(rng.integers(0, size, size // 3))}[present]
    else:  # sparse keys; -1 is the hash table's empty marker
        pool = np.concatenate([[-1], rng.integers(-2**62, 2**62, {"all": size // 2, "some": 37}[present])])
    k = rng.choice(pool, n).astype(np.int64)
    v = rng.integers(-2**40, 2**40, n)
    f = rng.standard_normal(n)
    e = q.Env()
    for t in (abi.T_I64, abi.T_I64, abi.T_F64):
        e.column(t)
    aggs = [q.Agg("COUNT"), q.Agg("SUM", q.col(1), "BIGINT", True), q.Agg("MIN", q.col(1), "BIGINT", True),
            q.Agg("MAX", q.col(2), "DOUBLE", True)]
    where = q.col(1).gt(2**50) if present == "none" else None
    aq = q.AggQuery(e, where, [(q.col(0), True)], aggs)
    ds = None
    if dense:
        ds = abi.DenseSpec()
        ds.G, ds.range[0], ds.stride[0] = size, size, 1
    bufs = [ops.DeviceBuffer.from_array(x) for x in (k, v, f)]
    views = [abi.ColView(b.ptr, t, 0, 0, 0) for b, t in zip(bufs, (abi.T_I64, abi.T_I64, abi.T_F64))]
    if present == "none":
        want = [np.zeros(0, np.int64)] * 4 + [np.zeros(0)]
    else:
        want = expected(k, v, f)
    ops.jit_set_mode(abi.JIT_SYNC)
    prog = ops.jit_get(e.env, e.ncols, aq.plan, abi.JF_DENSE if dense else abi.JF_GROUPED)
    ops.jit_set_mode(-1)
    agg = ops.GpuAggregator(aq.plan, size, ds)
    agg.add_batches(e.ncols, [(n, 0, views)])
    agg.run(e.env, prog)
    slots = [a.slot for a in aggs]

    def check(keys, exact):
        o = np.argsort(keys)
        assert np.array_equal(keys[o], want[0])
        x = exact[o]
        assert np.array_equal(x[:, slots[0], 0], want[1])
        assert np.array_equal(x[:, slots[1], 0], want[2]) and np.array_equal(x[:, slots[1], 1], want[2] >> 63)
        assert np.array_equal(x[:, slots[2], 0], want[3])
        assert np.array_equal(np.ascontiguousarray(x[:, slots[3], 0]).view(np.float64), want[4])

    # one-sync form, in ranges that split and pass the end
    g = want[0].size
    got_k, got_x = [], []
    step = max(1, g // 3 + 1)
    st = ops.HostBuffer(1, ops.FETCH_STATUS)
    hk, hx = ops.HostBuffer((step, 1), np.float64), ops.HostBuffer((step, aq.plan.naggs, 2), np.int64)
    for first in range(0, g + step, step):
        agg.fetch_async(step, hk, hx, st, first)
        ops.sync()
        assert st.array[0]["groups"] == g and not st.array[0]["overflow"] and not st.array[0]["error"]
        m = max(0, min(step, g - first))
        got_k.append(hk.array[:m, 0].view(np.int64).copy())
        got_x.append(hx.array[:m].copy())
    check(np.concatenate(got_k), np.concatenate(got_x))
    assert not agg.overflowed()
    keys, accs, exact = agg.fetch()
    check(keys[:, 0].view(np.int64), exact)
    if dense:
        assert np.array_equal(keys[:, 0].view(np.int64), want[0])  # ascending
        assert agg.group_count() == g
    kp, ap, cg = agg.compact()
    assert cg == g
    ck = ops.device_to_array(kp, np.int64, g)
    ca = ops.device_to_array(ap, np.int64, g * aq.plan.naggs).reshape(aq.plan.naggs, g)
    ops.tmp_free(kp)
    ops.tmp_free(ap)
    assert np.array_equal(ck, keys[:, 0].view(np.int64))
    assert np.array_equal(ca.T, accs.view(np.int64))
    agg.close()
