"""GPU: the VARCHAR page writer against the oracle: string lengths around
the widths of its copies, pages cut at their last byte, tiles of every size,
NULLs, and long strings between short ones."""
import numpy as np
import pytest

from calamarijoins_b200 import ColumnarTable, DataType, Plan, _lib, encode_column
from tests.helpers import assert_same, run_oracle, run_product

pytestmark = pytest.mark.gpu
I, V = DataType.INT32, DataType.VARCHAR


def _strings(kind, n, rng):
    lens = {"short": lambda: rng.integers(0, 9, n), "edges": lambda: rng.choice([0, 1, 3, 4, 5, 31, 32, 33, 255, 256, 257], n),
            "one_a_page": lambda: rng.integers(8100, 8186, n), "halves": lambda: rng.integers(4080, 4092, n),
            "empty": lambda: np.zeros(n, int),
            "long": lambda: np.where(rng.random(n) < 0.02, rng.integers(8186, 40_000, n), rng.integers(0, 60, n))}[kind]()
    pool = rng.integers(97, 123, 40_000).astype(np.uint8).tobytes()
    return [pool[i % 97:i % 97 + int(k)] for i, k in enumerate(lens)]


@pytest.mark.parametrize("tile_rows", [64, 2048, 8192])
@pytest.mark.parametrize("kind", ["short", "edges", "one_a_page", "halves", "empty", "long"])
@pytest.mark.parametrize("n", [1, 255, 2047, 2049, 9000])
def test_pages(gpu_ctx, tile_rows, kind, n):
    """A join that passes every row on, in several VARCHAR columns."""
    if kind in ("one_a_page", "halves", "long"):
        n = min(n, 2049)
    rng = np.random.default_rng(n)
    keys = np.arange(n, dtype=np.int32)
    some = (rng.random(n) > 0.3).astype(np.uint8)
    none = np.zeros(n, np.uint8)
    a = [encode_column(I, keys), encode_column(V, _strings(kind, n, rng)), encode_column(V, _strings(kind, n, rng), some)]
    b = [encode_column(I, rng.permutation(keys)), encode_column(V, _strings(kind, n, rng), none)]
    plan = Plan()
    plan.inputs = [ColumnarTable(n, a), ColumnarTable(n, b)]
    plan.new_scan_node(0, [(0, I), (1, V), (2, V)])
    plan.new_scan_node(1, [(0, I), (1, V)])
    plan.root = plan.new_join_node(True, 0, 1, 0, 0, [(0, I), (1, V), (2, V), (4, V)])
    want = run_oracle(plan)
    default = gpu_ctx.get_option(_lib.CJ_OPT_VARCHAR_TILE_ROWS)
    try:
        gpu_ctx.set_option(_lib.CJ_OPT_VARCHAR_TILE_ROWS, tile_rows)
        for flags in (0, _lib.CJ_EXEC_RESULT_ON_DEVICE):
            got, _ = run_product(plan, gpu_ctx, flags)
            assert_same(got, want, f"{kind} {n} rows")
    finally:
        gpu_ctx.set_option(_lib.CJ_OPT_VARCHAR_TILE_ROWS, default)
