"""What a new query shape compiles (no GPU: NVRTC targets sm_100a): kernels for batches stored otherwise than hinted and staged
kernels are not part of a plan's module, the hash scan holds one copy of its insertion per place, and the register
bounds follow the plan's width."""
import os
import re
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = r"""
import sys
from warpstore_b200 import abi, ops
from warpstore_b200 import query as q
kind, sums, enc = sys.argv[1], int(sys.argv[2]), int(sys.argv[3])
e = q.Env()
e.column(abi.T_I32, 0, enc)
for i in range(8):
    e.column(abi.T_I64, 0, enc)
aggs = [q.Agg("COUNT")] + [q.Agg("SUM", q.col(1 + i % 8) if i < 8 else q.col(1 + i % 8) + q.ilit(i), "BIGINT", i < 8)
                           for i in range(sums)]
aq = q.AggQuery(e, q.col(1).lt(500), [(q.col(0), True)], aggs)
fn = abi.JF_GROUPED if kind == "hash" else abi.JF_DENSE
print("SIZE", ops.codegen_compile_check(e.env, e.ncols, aq.plan, fn))
"""


def compiled(kind, sums, enc):
    env = dict(os.environ, WARPSTORE_B200_JIT_VERBOSE="1", PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD, kind, str(sums), str(enc)], env=env, cwd=ROOT, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    size = int(re.search(r"SIZE (\d+)", r.stdout)[1])
    spills = {m[1]: int(m[2]) for m in re.finditer(
        r"Compiling entry function '(\w+)'.*?\n.*?\n\D*\d+ bytes stack frame, (\d+) bytes spill stores", r.stderr)}
    return size, spills


def test_encoded_columns_do_not_double_the_module(built):
    raw, names = compiled("hash", 4, 0)
    enc, names_enc = compiled("hash", 4, 2)
    assert set(names) == set(names_enc) == {"wsq_hash", "wsq_multi_hash"}
    assert enc < 1.4 * raw, (raw, enc)


def test_dense_module_has_no_staged_kernels(built):
    _, names = compiled("dense", 4, 1)
    assert names and not any("staged" in n or n.startswith("wsg_") for n in names), names


@pytest.mark.parametrize("sums,limit", [(7, 400), (16, 500), (25, 1200)])
def test_register_bounds_follow_the_width(built, sums, limit):
    """Spill stores of the single-query hash scan (25 SUMs under the bound of narrow plans: over 5000 bytes)."""
    _, spills = compiled("hash", sums, 0)
    assert spills["wsq_hash"] <= limit, spills
