"""GPU: plans whose result is empty, or may be, against the oracle: columns
that no join gets to are not decoded."""
import numpy as np
import pytest

from calamarijoins_b200 import ColumnarTable, DataType, Plan, ResidentTable, _lib, encode_column
from tests.helpers import assert_same, run_oracle, run_product

pytestmark = pytest.mark.gpu
I, L, F = DataType.INT32, DataType.INT64, DataType.FP64


def _run(plan, ctx, resident, flags):
    """(result, launches by kernel) over resident tables or host pages."""
    rp = Plan()
    rp.nodes, rp.root = plan.nodes, plan.root
    rp.inputs = [ResidentTable(ctx, t) for t in plan.inputs] if resident else plan.inputs
    ctx.set_option(_lib.CJ_OPT_PROFILE_KERNELS, 1)
    ctx.profile_reset()
    try:
        got, _ = run_product(rp, ctx, flags)
        return got, {k: n for k, (n, _) in ctx.profile().items()}
    finally:
        ctx.set_option(_lib.CJ_OPT_PROFILE_KERNELS, 0)
        if resident:
            for t in rp.inputs:
                t.free()


def _fact(n, rng):
    ok = (rng.random(n) > 0.1).astype(np.uint8)
    return ColumnarTable(n, [encode_column(I, rng.integers(0, 500, n).astype(np.int32), ok),
                             encode_column(I, rng.integers(0, 500, n).astype(np.int32), ok),
                             encode_column(F, rng.random(n), ok), encode_column(L, np.arange(n), ok)])


def _dim(first, n=500):
    return ColumnarTable(n, [encode_column(I, np.arange(first, first + n, dtype=np.int32)),
                             encode_column(L, np.arange(n) * 7)])


@pytest.mark.parametrize("flags", [0, _lib.CJ_EXEC_RESULT_ON_DEVICE])
@pytest.mark.parametrize("resident", [True, False])
@pytest.mark.parametrize("empty", [0, 1, 2])
def test_empty_table(gpu_ctx, empty, resident, flags):
    """Two joins; one of the three tables has no rows."""
    rng = np.random.default_rng(1)
    plan = Plan()
    plan.inputs = [_fact(0 if empty == 0 else 20_000, rng), _dim(0, 0 if empty == 1 else 500), _dim(0, 0 if empty == 2 else 500)]
    fact = plan.new_scan_node(0, [(0, I), (1, I), (2, F), (3, L)])
    dims = [plan.new_scan_node(k, [(0, I), (1, L)]) for k in (1, 2)]
    j = plan.new_join_node(True, fact, dims[0], 0, 0, [(1, I), (2, F), (3, L), (5, L)])
    plan.root = plan.new_join_node(True, j, dims[1], 0, 0, [(1, F), (2, L), (3, L), (5, L)])
    got, launches = _run(plan, gpu_ctx, resident, flags)
    assert_same(got, run_oracle(plan))
    assert got.num_rows == 0
    if empty < 2:  # the first join: nothing is read at all
        assert "decode" not in launches and "page_index" not in launches


@pytest.mark.parametrize("flags", [0, _lib.CJ_EXEC_RESULT_ON_DEVICE])
@pytest.mark.parametrize("first", [0, 1000])
@pytest.mark.parametrize("n", [20_000, 19_000_000])
def test_empty_join(gpu_ctx, first, n, flags):
    """The first join matches something or nothing: payloads of more than 256
    MB of pages are decoded (the second launch) only when the root is
    reached."""
    rng = np.random.default_rng(2)
    plan = Plan()
    plan.inputs = [_fact(n, rng), _dim(first), _dim(0, 5)]
    fact = plan.new_scan_node(0, [(0, I), (1, I), (2, F), (3, L)])
    dims = [plan.new_scan_node(k, [(0, I), (1, L)]) for k in (1, 2)]
    j = plan.new_join_node(True, fact, dims[0], 0, 0, [(1, I), (2, F), (3, L), (5, L)])
    plan.root = plan.new_join_node(True, j, dims[1], 0, 0, [(1, F), (2, L), (3, L), (5, L)])
    got, launches = _run(plan, gpu_ctx, True, flags)
    assert_same(got, run_oracle(plan))
    assert (got.num_rows == 0) == (first > 0)
    assert launches["decode"] == (2 if n > 20_000 and not first else 1)
    assert launches["page_index"] == 1
