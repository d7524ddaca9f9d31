"""ws_gather_multi over every storage: encodings 1-6 with NULLs, batches that mix raw and encoded storage, empty batches,
and more batches than their offsets fit in shared memory."""
import numpy as np
import pytest

from warpstore_b200 import abi, ops
from warpstore_b200 import workloads as W

from .test_decimal_scans_gpu import segment

pytestmark = pytest.mark.gpu


def stored(values, enc, null):
    """(bytes, what a gather gives) of one batch."""
    if enc == 0:
        return np.ascontiguousarray(values).view(np.uint8), values
    if enc <= 3:
        return W.encode_for(values, {1: 1, 2: 2, 3: 4}[enc], null)[0], values
    rng = np.random.default_rng(values.size)
    top = {4: 256, 5: 65535, 6: 2**32 - 1}[enc]
    codes = rng.integers(0, top, values.size)
    if enc == 4:
        d = rng.standard_normal(256)
        return segment(codes, 4, 0, 0, d), d[codes]
    codes[::7] = top
    out = (codes.astype(np.int64) - 900) / 100.0
    out[::7] = np.nan
    return segment(codes, enc, -900, 100.0), out


@pytest.mark.parametrize("ptype,encs", [(abi.PT_I64, (1,)), (abi.PT_I64, (3, 0, 1, 2)), (abi.PT_I32, (1, 0)), (abi.PT_I32, (2,)),
                                        (abi.PT_F64, (4,)), (abi.PT_F64, (5, 0)), (abi.PT_F64, (6, 4, 5, 0)), (abi.PT_F64, (0,))])
@pytest.mark.parametrize("sizes", [[1], [5, 0, 4097, 0, 0, 1023, 0], [3, 1, 2] * 900])
def test_storages(ptype, encs, sizes):
    rng = np.random.default_rng(len(sizes))
    dt, null = {abi.PT_I64: (np.int64, abi.NULL_I64), abi.PT_I32: (np.int32, abi.NULL_I32), abi.PT_F64: (np.float64, None)}[ptype]
    raw, want, at = [], [], 0
    offs, boff = [], []
    for b, n in enumerate(sizes):
        v = rng.integers(-90, 90, n).astype(dt)
        if null is not None:
            v[rng.random(n) < 0.1] = null
        enc = encs[b % len(encs)]
        s, w = stored(v, enc, null)
        raw.append(s), want.append(w), boff.append(at)
        at += n
    starts = np.concatenate([[0], np.cumsum([(s.size + 255) // 256 * 256 for s in raw])])
    host = np.zeros(int(starts[-1]) + 256, np.uint8)
    for s, o in zip(raw, starts):
        host[o:o + s.size] = s
    dev = ops.DeviceBuffer.from_array(host)
    t = {abi.PT_I64: abi.T_I64N, abi.PT_I32: abi.T_I32N, abi.PT_F64: abi.T_F64}[ptype]
    views = [abi.ColView(dev.ptr + int(o), t, 0, encs[b % len(encs)], 0) for b, o in enumerate(starts[:-1])]
    want = np.concatenate(want).astype(dt)
    for idx in (np.arange(at), np.arange(at)[::-1], rng.integers(0, at, 2049)):
        di = ops.DeviceBuffer.from_array(idx.astype(np.int32))
        out = ops.DeviceBuffer(idx.size * dt().itemsize + 16)
        ops.gather_multi(views, boff, ptype, dt().itemsize, di.ptr, idx.size, out.ptr)
        np.testing.assert_array_equal(out.to_array(dt, idx.size), want[idx])
