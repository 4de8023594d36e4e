"""GPU: probes of repeated keys with several matches a row, against the
oracle: matches per row on both sides of what the probe packs (3), of its
buffer (320) and of a warp, mixed in one page, by one block per step of the
probe side and by two, four and eight (few probe rows)."""
import numpy as np
import pytest

from calamarijoins_b200 import ColumnarTable, DataType, Plan, ResidentTable, _lib, encode_column
from tests.helpers import assert_same, run_oracle, run_product
from tests.test_gpu_unique import _check, _plan

pytestmark = pytest.mark.gpu
I, L, F = DataType.INT32, DataType.INT64, DataType.FP64


def _build(rng, counts, gap):
    """Keys with these numbers of rows each, in a random order."""
    keys = rng.permutation(len(counts)) * gap
    return keys, rng.permutation(np.repeat(keys, counts))


@pytest.mark.parametrize("counts", [[1, 2, 3, 4, 5, 31, 32, 33, 40], [2, 3], [3, 3, 3, 4], [319, 320, 321, 2, 1], [5]])
@pytest.mark.parametrize("kt,gap", [(I, 1), (I, 10 ** 5), (L, 1), (L, 10 ** 12)])
def test_matches_per_row(gpu_ctx, kt, gap, counts):
    rng = np.random.default_rng(len(counts))
    keys, bkeys = _build(rng, counts * (40 if max(counts) < 300 else 2), gap)
    n = 4 * len(bkeys) + 3000
    pkeys = keys[rng.integers(0, len(keys), n)] + (rng.random(n) < 0.6) * gap * 1000
    pok = (rng.random(n) >= 0.05).astype(np.uint8)
    plan = _plan(bkeys, pkeys, kt, kt, None, pok, bpay=[(L, np.arange(len(bkeys)), None)],
                 ppay=[(F, np.arange(n) / 4, None)])
    _check(plan, gpu_ctx, "hash")


@pytest.mark.parametrize("gap", [1, 1000])
@pytest.mark.parametrize("n", [3000, 600_000, 1_100_000, 2_600_000])
def test_blocks_per_step(gpu_ctx, n, gap):
    """Eight, four and two blocks for a page of probe rows, and one."""
    rng = np.random.default_rng(n)
    keys, bkeys = _build(rng, [1, 2, 3, 4, 9, 40, 330] * 6, gap)
    pkeys = np.full(n, -5)
    hit = rng.permutation(n)[:3000]
    pkeys[hit] = keys[rng.integers(0, len(keys), 3000)]
    pok = (rng.random(n) >= 0.02).astype(np.uint8)
    plan = _plan(bkeys, pkeys, pvalid=pok, bpay=[(L, np.arange(len(bkeys)), None)], ppay=[(I, np.arange(n), None)])
    want = run_oracle(plan)
    got, st = run_product(plan, gpu_ctx)
    assert_same(got, want, f"{n} probe rows")


def _resident_run(plan, ctx, flags=0):
    rp = Plan()
    rp.nodes, rp.root = plan.nodes, plan.root
    rp.inputs = [ResidentTable(ctx, t) for t in plan.inputs]
    try:
        return run_product(rp, ctx, flags)[0]
    finally:
        for t in rp.inputs:
            t.free()


@pytest.mark.parametrize("pay", ["dense", "nulls"])
@pytest.mark.parametrize("kt,pt,gap", [(I, I, 1), (I, L, 10 ** 5), (L, L, 1), (L, I, 1000)])
@pytest.mark.parametrize("counts", [[63, 64, 65], [959, 960, 961, 1], [1919, 1920, 1921, 4, 5], [5000, 63, 2], [64]])
def test_runs(gpu_ctx, counts, kt, pt, gap, pay):
    """Matches that a kernel of their own writes (64 a row or more, 960 a
    run), beside rows of fewer: into pages and, with NULLs, as row ids."""
    rng = np.random.default_rng(len(counts))
    keys, bkeys = _build(rng, counts * 3, gap)
    bkeys -= gap  # a negative key too
    n = max(4 * len(bkeys), 65_536)  # room for fewer: the probe writes them itself
    pkeys = np.full(n, 10 ** 8)
    hit = rng.permutation(n)[:40]
    pkeys[hit] = keys[rng.integers(0, len(keys), 40)] - gap
    ok = (lambda rows: (rng.random(rows) >= 0.2).astype(np.uint8)) if pay == "nulls" else (lambda rows: None)
    plan = _plan(bkeys, pkeys, kt, pt, pvalid=(rng.random(n) >= 0.02).astype(np.uint8),
                 bpay=[(L, np.arange(len(bkeys)), ok(len(bkeys))), (I, np.arange(len(bkeys)), None)],
                 ppay=[(F, np.arange(n) / 4, ok(n)), (I, np.arange(n), None)])
    want = run_oracle(plan)
    for flags in (0, _lib.CJ_EXEC_RESULT_ON_DEVICE):
        assert_same(_resident_run(plan, gpu_ctx, flags), want, f"{counts}")


@pytest.mark.parametrize("gap", [1, 10 ** 5])
def test_runs_below_the_root(gpu_ctx, gap):
    """Runs of an intermediate's row ids, and of a probe side and a build side
    that are intermediates."""
    rng = np.random.default_rng(3)
    keys, bkeys = _build(rng, [1, 70, 1000, 3], gap)
    many = ColumnarTable(len(bkeys), [encode_column(I, bkeys.astype(np.int32)), encode_column(L, np.arange(len(bkeys)))])
    n = 100_000
    fk = np.where(rng.random(n) < 0.005, keys[rng.integers(0, len(keys), n)], -9)
    fact = ColumnarTable(n, [encode_column(I, np.arange(n, dtype=np.int32)), encode_column(I, fk.astype(np.int32)),
                             encode_column(F, rng.random(n))])
    ids = rng.permutation(n)[:95_000]
    some = ColumnarTable(95_000, [encode_column(I, ids.astype(np.int32)), encode_column(I, (ids * 3).astype(np.int32))])
    plan = Plan()
    plan.inputs = [many, fact, some]
    s = [plan.new_scan_node(0, [(0, I), (1, L)]), plan.new_scan_node(1, [(0, I), (1, I), (2, F)]),
         plan.new_scan_node(2, [(0, I), (1, I)])]
    j = plan.new_join_node(True, s[0], s[1], 0, 1, [(2, I), (1, L), (3, I), (4, F)])  # below the root
    plan.root = plan.new_join_node(True, j, s[2], 0, 0, [(0, I), (1, L), (2, I), (3, F), (5, I)])
    assert_same(_resident_run(plan, gpu_ctx), run_oracle(plan), "below")
    plan = Plan()
    plan.inputs = [many, fact, some]
    s = [plan.new_scan_node(0, [(0, I), (1, L)]), plan.new_scan_node(1, [(0, I), (1, I), (2, F)]),
         plan.new_scan_node(2, [(0, I), (1, I)])]
    j = plan.new_join_node(True, s[1], s[2], 0, 0, [(1, I), (2, F), (4, I)])
    plan.root = plan.new_join_node(True, s[0], j, 0, 0, [(0, I), (1, L), (2, I), (3, F), (4, I)])
    assert_same(_resident_run(plan, gpu_ctx), run_oracle(plan), "probe side")


@pytest.mark.parametrize("pt", [I, L])
def test_runs_of_dense_keys(gpu_ctx, pt):
    """The host does not know the longest run of dense keys: from 1M rows of
    room on."""
    rng = np.random.default_rng(8)
    keys, bkeys = _build(rng, [64, 63, 961, 3, 1, 1920], 1)
    n = 1 << 20
    pkeys = np.full(n, 10 ** 8)
    hit = rng.permutation(n)[:200]
    pkeys[hit] = keys[rng.integers(0, len(keys), 200)]
    plan = _plan(bkeys, pkeys, I, pt, bpay=[(L, np.arange(len(bkeys)), None)], ppay=[(I, np.arange(n), None)])
    assert_same(_resident_run(plan, gpu_ctx, _lib.CJ_EXEC_RESULT_ON_DEVICE), run_oracle(plan))
