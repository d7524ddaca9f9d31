"""Memory of large result tables: kept for the next query up to the table pool's bound and beyond it, and given back when
asked for."""
import pytest

from warpstore_b200 import abi, ops
from warpstore_b200 import query as q
from warpstore_b200._lib import lib

pytestmark = pytest.mark.gpu
GB = 1 << 30


def table(cap, fns):
    e = q.Env()
    e.column(abi.T_I64, 0, 0)
    aq = q.AggQuery(e, None, [(q.col(0), True)], [q.Agg("COUNT")] + [q.Agg(f, q.col(0), "BIGINT", True) for f in fns])
    return ops.GpuAggregator(aq.plan, cap)


def free_memory():
    ops.sync()
    return int(lib().ws_vram_free())


@pytest.fixture(autouse=True)
def trimmed():
    lib().ws_gpu_trim_pool()
    yield
    lib().ws_gpu_trim_pool()


def test_tables_past_the_bound_stay_mapped():
    before = free_memory()
    a = table(1 << 29, ("SUM", "MIN", "MAX"))  # 26 GB: more than an eighth of 180 GB
    used = before - free_memory()
    assert used > 20 * GB
    a.close()
    assert before - free_memory() > used - (64 << 20), "unmapped at a synchronisation"
    lib().ws_gpu_trim_pool()
    assert before - free_memory() < GB
