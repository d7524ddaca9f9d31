"""The double dictionary (enc 4) where its collection of distinct patterns can go wrong: the 255-pattern
limit, +0.0 as a pattern of its own, a pattern that only the last row has, columns of one tile and of many
CTAs — byte for byte against the oracle."""
import numpy as np
import pytest

from oracle import oracle
from warpstore_b200 import abi, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1024, 1025, 70_001, (1 << 20) + 3])
@pytest.mark.parametrize("distinct,zero,last", [(1, False, False), (254, True, False), (255, False, True),
                                                (255, True, True), (256, False, True), (5000, True, False)])
def test_dictionary_limits(n, distinct, zero, last):
    rng = np.random.default_rng(n + distinct)
    vals = rng.random(distinct) * 1e6 + 0.123456789
    x = rng.choice(vals[:-1] if last and distinct > 1 else vals, n)
    x[:min(distinct, n) - 1] = vals[:min(distinct, n) - 1]  # every pattern occurs ...
    if not last:
        x[rng.integers(0, n)] = vals[-1]
    if zero:
        x[n // 2] = 0.0
        x[n - 2] = -0.0
    if last:
        x[n - 1] = vals[-1]  # ... the last one only in the last row
    oe, ob = oracle.encode_column_engine(x, abi.PT_F64)
    d = ops.DeviceBuffer.from_array(x)
    ptr, nbytes, enc = ops.encode_column_engine(d.ptr, abi.PT_F64, n)
    assert enc == oe
    if enc:
        assert np.array_equal(ops.device_to_array(ptr, np.uint8, nbytes), ob)
        ops.tmp_free(ptr)
