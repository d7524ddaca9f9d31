"""ws_eval_at / ws_eval_at_int of arithmetic over raw columns (the register-stack form) at the edges of its
groups of rows and of its stack, with NULLs, division by zero and row indices, against the oracle; one deeper
program and an encoded column take the general form."""
import numpy as np
import pytest

from oracle import oracle
from warpstore_b200 import abi, ops
from warpstore_b200 import query as q
from warpstore_b200 import workloads as W

pytestmark = pytest.mark.gpu


def programs():
    c = [q.col(i) for i in range(6)]
    return [c[0], c[1], c[2], c[3], c[4], c[5], -c[1], -c[2], c[0] + c[1], c[1] * (q.ilit(100) - c[0]) / q.lit(100.0),
            c[2] / c[0], c[3] + c[4] * c[2], c[0] - (c[1] - (c[0] - c[1])), c[0] - (c[1] - (c[0] - (c[1] - c[0]))),
            c[5] * c[0], q.lit(2.5), q.ilit(7) - c[3]]


@pytest.mark.parametrize("n", [1, 255, 1024, 1025, 5003])
@pytest.mark.parametrize("with_idx", [False, True])
def test_eval_simple(n, with_idx):
    rng = np.random.default_rng(n)
    t = W.Table(n)
    t.add("a", abi.T_I32, rng.integers(-3, 4, n).astype(np.int32))
    t.add("b", abi.T_I64, rng.integers(-10**9, 10**9, n))
    t.add("c", abi.T_F64, np.where(rng.random(n) < 0.2, np.nan, rng.standard_normal(n)))
    t.add("d", abi.T_I32N, np.where(rng.random(n) < 0.2, abi.NULL_I32, rng.integers(0, 9, n)).astype(np.int32))
    t.add("e", abi.T_I64N, np.where(rng.random(n) < 0.2, abi.NULL_I64, rng.integers(0, 9, n)))
    t.add("f", abi.T_I64, rng.integers(0, 200, n), enc=1)
    t.to_device()
    e = W.env_for(t)
    for i, v in enumerate(t.views(0, True)):
        e.env.cols[i] = v
    idx = rng.integers(0, n, 2 * n + 1).astype(np.int32) if with_idx else None
    m = idx.size if with_idx else n
    di = ops.DeviceBuffer.from_array(idx) if with_idx else None
    out = ops.DeviceBuffer(m * 8)
    for x in programs():
        prog = e.compile(x)
        for as_int in (False, True):
            (ops.eval_at_int if as_int else ops.eval_at)(e.env, e.ncols, prog, di.ptr if di else None, m, out.ptr)
            want, _ = oracle.eval_at(e.env, t.views(0, False), prog, idx, m, as_int)
            got = out.to_array(np.int64 if as_int else np.float64, m)
            assert np.array_equal(got, want, equal_nan=not as_int)
    t.free_device()
