"""GPU: the page index and decode of all of a plan's columns in one launch
each, against the oracle: page counts around the index's chunk of 256, more
columns than one launch takes (32) and than the status block tracks (64),
and columns whose errors must not count until the plan reads them."""
import numpy as np
import pytest

from calamarijoins_b200 import CJError, Column, ColumnarTable, DataType, Plan, ResidentTable, _lib, encode_column
from tests.helpers import assert_same, run_oracle, run_product

pytestmark = pytest.mark.gpu
I, L, F, V = DataType.INT32, DataType.INT64, DataType.FP64, DataType.VARCHAR


def _run_resident(plan, ctx, flags=_lib.CJ_EXEC_RESULT_ON_DEVICE):
    rp = Plan()
    rp.nodes, rp.root = plan.nodes, plan.root
    rp.inputs = [ResidentTable(ctx, t) for t in plan.inputs]
    try:
        return run_product(rp, ctx, flags)[0]
    finally:
        for t in rp.inputs:
            t.free()


def _scan(columns, rows):
    plan = Plan()
    plan.inputs.append(ColumnarTable(rows, columns))
    plan.root = plan.new_scan_node(0, [(i, c.type) for i, c in enumerate(columns)])
    return plan


@pytest.mark.parametrize("pages", [1, 255, 256, 257, 600])
def test_index_chunks(gpu_ctx, pages):
    rng = np.random.default_rng(pages)
    n = pages * 1984 - 7
    valid = (rng.random(n) > 0.1).astype(np.uint8)
    cols = [encode_column(I, np.arange(n, dtype=np.int32)),
            encode_column(I, rng.integers(0, 1000, n).astype(np.int32), valid),
            encode_column(L, rng.integers(0, 1 << 50, n), valid)]
    plan = _scan(cols, n)
    for flags in (0, _lib.CJ_EXEC_RESULT_ON_DEVICE):
        got = _run_resident(plan, gpu_ctx, flags)
        assert_same(got, run_oracle(plan), f"{pages} pages")


@pytest.mark.parametrize("ncols", [31, 32, 33, 64, 70])
def test_many_columns(gpu_ctx, ncols):
    rng = np.random.default_rng(ncols)
    n = 3000
    cols = []
    for c in range(ncols):
        valid = (rng.random(n) > 0.2).astype(np.uint8) if c % 3 == 1 else None
        t = (I, L, F, V)[c % 4]
        if t == V:
            cols.append(encode_column(V, ["s%d" % x for x in rng.integers(0, 10 ** 6, n)], valid))
        else:
            cols.append(encode_column(t, rng.integers(0, 10 ** 6, n), valid))
    plan = _scan(cols, n)
    got = _run_resident(plan, gpu_ctx)
    assert_same(got, run_oracle(plan), f"{ncols} columns")


@pytest.mark.parametrize("empty", [True, False])
def test_errors_of_unread_columns(gpu_ctx, empty):
    """The payload of the last table has a page with more values than rows:
    rejected when the plan reads the column, accepted when the join below is
    empty and nothing reads it."""
    n = 5000
    a = ColumnarTable(n, [encode_column(I, np.arange(n, dtype=np.int32))])
    b = ColumnarTable(n, [encode_column(I, np.arange(n, dtype=np.int32) + (10 * n if empty else 0))])
    bad = encode_column(I, np.arange(n, dtype=np.int32)).pages.copy()
    bad[0, 2] = 0xFF
    bad[0, 3] = 0x7F
    c = ColumnarTable(n, [encode_column(I, np.arange(n, dtype=np.int32)), Column(I, bad)])
    plan = Plan()
    plan.inputs = [a, b, c]
    s = [plan.new_scan_node(0, [(0, I)]), plan.new_scan_node(1, [(0, I)]), plan.new_scan_node(2, [(0, I), (1, I)])]
    j = plan.new_join_node(True, s[0], s[1], 0, 0, [(0, I)])
    plan.root = plan.new_join_node(True, j, s[2], 0, 0, [(0, I), (2, I)])
    if empty:
        assert _run_resident(plan, gpu_ctx).num_rows == 0
    else:
        with pytest.raises(CJError) as ei:
            _run_resident(plan, gpu_ctx)
        assert ei.value.status == 3
    plan.inputs[2] = ColumnarTable(n, [c.columns[0], c.columns[0]])
    got = _run_resident(plan, gpu_ctx)
    assert got.num_rows == (0 if empty else n)  # the context is as usable as before
