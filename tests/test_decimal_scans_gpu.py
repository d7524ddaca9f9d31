"""Compiled scans over dictionary and decimal segments (encodings 4-6): the scan's quotient (a multiplication by the
reciprocal, corrected) equals the division bit for bit over every scale and base it accepts and on both sides of its
fallback, NULL codes and ragged, unaligned batches included, against the CPU oracle's division."""
import numpy as np
import pytest

from oracle import oracle
from warpstore_b200 import abi, ops
from warpstore_b200 import query as q

from .helpers import compare_exact

pytestmark = pytest.mark.gpu
EDGE = 1 << 51  # |base| below it takes the reciprocal


def segment(codes, enc, base, p10, dictionary=None):
    """The stored bytes: int64 base, double 10^scale, the dictionary (enc 4), the codes, 16 pad bytes."""
    head = np.int64(base).tobytes() + np.float64(p10).tobytes() if enc != 4 else bytes(16)
    body = (dictionary.tobytes() if enc == 4 else b"") + codes.astype({4: np.uint8, 5: np.uint16, 6: np.uint32}[enc]).tobytes()
    return np.frombuffer(head + body + bytes(16), np.uint8)


def run(kind, segs, enc, cut, offs):
    e = q.Env()
    e.column(abi.T_F64, 0, enc)
    e.column(abi.T_I32, 0, 0)
    aggs = [q.Agg("COUNT"), q.Agg("MIN", q.col(0), "DOUBLE", True), q.Agg("MAX", q.col(0), "DOUBLE", True)]
    aq = q.AggQuery(e, q.col(0).lt(cut) if cut is not None else None, {"value": [(q.col(0), False)], "nokeys": [],
                                                                       "row": [(q.col(1), True)]}[kind], aggs)
    ops.jit_set_mode(abi.JIT_SYNC)
    try:
        prog = ops.jit_get(e.env, e.ncols, aq.plan, abi.JF_NOKEYS if kind == "nokeys" else abi.JF_GROUPED, "test")
    finally:
        ops.jit_set_mode(-1)
    assert prog
    host, dev, keep, total = [], [], [], 0
    for (n, seg), off in zip(segs, offs):
        rows = np.arange(total, total + n, dtype=np.int32)
        d, r = ops.DeviceBuffer.from_array(seg), ops.DeviceBuffer.from_array(rows)
        keep += [seg, d, rows, r]
        host.append((n, 0, [abi.ColView(seg.ctypes.data, abi.T_F64, 0, enc, off), abi.ColView(rows.ctypes.data, abi.T_I32, 0, 0, 0)]))
        dev.append((n, 0, [abi.ColView(d.ptr, abi.T_F64, 0, enc, off), abi.ColView(r.ptr, abi.T_I32, 0, 0, 0)]))
        total += n
    ok, ow, _ = oracle.aggregate(e.env, aq.plan, host, e.ncols)
    agg = ops.GpuAggregator(aq.plan, 1 << (2 * total - 1).bit_length())
    agg.add_batches(e.ncols, dev)
    agg.run(e.env, prog)
    assert not agg.overflowed()
    k, _, x = agg.fetch()
    compare_exact(aq.plan, k, x, ok, ow)
    agg.close()


@pytest.mark.parametrize("kind", ["value", "nokeys", "row"])
@pytest.mark.parametrize("enc,base,p10", [(5, b, 10.0 ** s) for s in range(5) for b in (0, -70_001)] +
                         [(6, b, p) for p in (1.0, 100.0, 10_000.0, 1e15, 1e16) for b in
                          (-EDGE, -EDGE + 1, EDGE - 1, EDGE, -(1 << 31), 123_456_789_012)])
def test_decimals(enc, base, p10, kind):
    rng = np.random.default_rng(abs(base) % 1000 + int(np.log10(p10)))
    top = (1 << (16 if enc == 5 else 32)) - 1
    segs, offs = [], []
    for n, off in ((4096, 0), (1023, 3), (1, 0), (2051, 1)):  # ragged; views that start inside a segment
        codes = rng.integers(0, top, n + off)
        codes[rng.random(n + off) < 0.1] = top  # NULL
        codes[:2] = [0, top - 1][:codes[:2].size]
        segs.append((n, segment(codes, enc, base, p10)))
        offs.append(off)
    run(kind, segs, enc, None if kind == "row" else (base + top // 2) / p10, offs)


@pytest.mark.parametrize("kind", ["value", "nokeys", "row"])
def test_dictionaries(kind):
    rng = np.random.default_rng(5)
    values = np.concatenate([rng.standard_normal(250) * 10.0 ** rng.integers(-200, 200, 250), [0.0, 1e308, 5e-324, np.nan, 1, 2]])
    segs, offs = [], []
    for n, off in ((4096, 0), (1023, 3), (5, 1)):
        segs.append((n, segment(rng.integers(0, 256, n + off), 4, 0, 0, rng.permutation(values))))
        offs.append(off)
    run(kind, segs, 4, 1e300, offs)
