"""ws_sort_perm at the edges of its radix sort: tile boundaries, one row, composites of at most 32, at most
64 and several 64-bit words, constant keys, NULL (NaN), infinities and signed zeros, ties (stability),
descending keys — against the oracle's stable sort."""
import numpy as np
import pytest

from oracle import oracle
from warpstore_b200 import ops

pytestmark = pytest.mark.gpu


def key(kind, n, rng):
    if kind == "const":
        return np.full(n, 42.0)
    if kind == "few":  # many ties
        return rng.integers(0, 3, n).astype(np.float64)
    if kind == "date":
        return rng.integers(8000, 10557, n).astype(np.float64)
    if kind == "wide":  # every bit of the order key varies
        return rng.standard_normal(n) * np.exp(rng.uniform(-600, 600, n))
    x = rng.standard_normal(n)  # "special"
    x[rng.random(n) < 0.3] = np.nan
    for v in (np.inf, -np.inf, 0.0, -0.0, 5e-324, -5e-324):
        x[rng.random(n) < 0.1] = v
    return x


@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 3 * 4096 + 5, 1_100_003])
@pytest.mark.parametrize("kinds,desc", [(("const",), (0,)), (("few", "const"), (1, 1)), (("date", "few"), (1, 0)),
                                        (("special",), (1,)), (("few", "special"), (0, 0)),
                                        (("few", "wide", "date", "wide"), (1, 0, 1, 1)),
                                        (("few",) * 11, (0, 1) * 5 + (1,)), ((), ())])
def test_sort_perm(n, kinds, desc):
    rng = np.random.default_rng(n * 31 + len(kinds))
    keys = [key(k, n, rng) for k in kinds]
    bufs = [ops.DeviceBuffer.from_array(k) for k in keys]
    perm = ops.sort_perm([b.ptr for b in bufs], list(desc), n)
    got = ops.device_to_array(perm, np.int32, n)
    ops.tmp_free(perm)
    want = oracle.sort_perm(keys, [bool(d) for d in desc]) if keys else np.arange(n, dtype=np.int32)
    assert np.array_equal(got, want)
