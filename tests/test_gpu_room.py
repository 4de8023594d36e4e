"""GPU: memory that a plan sets aside for matches that may not come, bounded
by CJ_SPARE_ROOM_BYTES, against the oracle: joins whose result columns the
probe may not write, or may write in its first run and not in the second."""
import numpy as np
import pytest

from calamarijoins_b200 import (CJError, ColumnarTable, Context, DataType, Plan, ResidentTable, Server, _lib,
                                encode_column, execute_batch, execute_raw)
from oracle import oracle_api as oa
from tests.helpers import assert_same, run_oracle, run_product
from tests.test_gpu_unique import _plan

pytestmark = pytest.mark.gpu
I, L, F, V = DataType.INT32, DataType.INT64, DataType.FP64, DataType.VARCHAR


def _resident(plan, ctx):
    rp = Plan()
    rp.nodes, rp.root = plan.nodes, plan.root
    rp.inputs = [ResidentTable(ctx, t) for t in plan.inputs]
    return rp


@pytest.fixture
def bounded(monkeypatch):
    """Runs a plan over resident tables in a context with a bound of its own
    on the room."""
    def run(plan, room, flags):
        monkeypatch.setenv("CJ_SPARE_ROOM_BYTES", str(room))
        ctx = Context(0)
        rp = _resident(plan, ctx)
        try:
            return run_product(rp, ctx, flags)
        finally:
            for t in rp.inputs:
                t.free()
            ctx.close()

    return run


@pytest.mark.parametrize("flags", [0, _lib.CJ_EXEC_RESULT_ON_DEVICE])
@pytest.mark.parametrize("gap", [1, 5000])
@pytest.mark.parametrize("room", [0, 600_000, 1_450_000, 1 << 30])
def test_room_refused(bounded, room, gap, flags):
    """Three build rows per key and 60,000 matches for 20,000 probe rows (and
    4,500 that match nothing): the payload columns' pages take 23 bytes a row,
    460 (564) KB for the probe rows and 1,380 KB for the matches, so that the
    bound refuses every run, the second one only (600,000), the pages of a
    first run with room for all (1,450,000) or nothing."""
    rng = np.random.default_rng(2)
    bkeys = rng.permutation(np.repeat(np.arange(2000) * gap, 3))
    n = 20_000 if gap == 1 else 24_500
    pkeys = np.concatenate([rng.integers(0, 2000, 20_000) * gap, np.full(n - 20_000, -7)])
    valid = (rng.random(len(bkeys)) >= 0.1).astype(np.uint8)
    plan = _plan(bkeys, rng.permutation(pkeys), bpay=[(L, np.arange(6000), None), (I, np.arange(6000), valid)],
                 ppay=[(F, rng.random(n), None)])
    got, st = bounded(plan, room, flags)
    assert_same(got, run_oracle(plan), f"room {room}")
    assert got.num_rows == 60_000
    if room == 0:
        assert st.exec["probe_reruns"] == 1


@pytest.mark.parametrize("gap", [1, 5000])
@pytest.mark.parametrize("rows", [5, 4])
def test_room_for_the_mean_is_enough(gpu_ctx, rows, gap):
    """Probe rows that all match, of keys with a row more than the mean a
    little more often than of the others: one run."""
    k = np.arange(4000) * gap
    bkeys = np.concatenate([np.repeat(k, rows - 3), k[:1000]])
    pkeys = np.concatenate([np.repeat(k, 12), k[:500]])
    plan = _plan(bkeys, pkeys, bpay=[(L, np.arange(len(bkeys)), None)])
    rp = _resident(plan, gpu_ctx)
    try:
        got, st = run_product(rp, gpu_ctx, _lib.CJ_EXEC_RESULT_ON_DEVICE)
    finally:
        for t in rp.inputs:
            t.free()
    assert_same(got, run_oracle(plan))
    assert got.num_rows > len(pkeys) * len(bkeys) // 4000
    assert st.exec["probe_reruns"] == 0


@pytest.mark.parametrize("gap", [1, 5000])
@pytest.mark.parametrize("room", [0, 1 << 30])
def test_device_counted_result(bounded, room, gap):
    """Unique keys, result in HBM: written with the count on the device (one
    synchronisation) only where the probe rows' pages may be set aside."""
    rng = np.random.default_rng(4)
    bkeys, n = rng.permutation(3000) * gap, 40_000
    pkeys = bkeys[rng.integers(0, 3000, n)] + gap * 3000 * (rng.random(n) < 0.9)
    plan = _plan(bkeys, pkeys, bpay=[(L, np.arange(3000), None)], ppay=[(F, rng.random(n), None)])
    got, st = bounded(plan, room, _lib.CJ_EXEC_RESULT_ON_DEVICE)
    assert_same(got, run_oracle(plan), f"room {room}")
    assert st.exec["host_syncs"] == (2 if room == 0 else 1)


@pytest.mark.parametrize("flags", [0, _lib.CJ_EXEC_RESULT_ON_DEVICE])
@pytest.mark.parametrize("keys", ["unique", "repeated"])
def test_selective_result_gives_room_back(gpu_ctx, keys, flags):
    """A handful of matches for 10M probe rows: the result holds the pages of
    its matches, not those of the matches there might have been (41 MB for the
    keys, 81 MB for each payload)."""
    nb, n = 3000, 10_000_000
    bkeys = np.arange(nb) if keys == "unique" else np.arange(nb) // 2
    pkeys = np.full(n, 10 ** 6)
    pkeys[::1_000_000] = 7
    plan = _plan(bkeys, pkeys, bpay=[(L, np.arange(nb), None)], ppay=[(F, np.arange(n) / 2, None)])
    rp = _resident(plan, gpu_ctx)
    gpu_ctx.set_option(_lib.CJ_OPT_BUFFER_CACHE_BYTES, 0)  # freed buffers go back to the pool at once
    try:
        before, _ = gpu_ctx.memory()
        res, _ = execute_raw(rp, gpu_ctx, flags)
        held = gpu_ctx.memory()[0] - before
        got = oa.PagedResult.from_result(res)
        res.free()
        assert held < 1 << 20
        assert_same(got, run_oracle(plan), keys)
    finally:
        gpu_ctx.set_option(_lib.CJ_OPT_BUFFER_CACHE_BYTES, 16 << 30)
        for t in rp.inputs:
            t.free()


@pytest.mark.parametrize("keys", ["dense", "spread", "wide", "repeated", "repeated_spread"])
def test_plan_does_without_spare_room(gpu_ctx, keys):
    """Every allocation of a join fails in turn. What the plan can do without
    (open-addressing slots, pages that the probe writes, room above the probe
    rows, tables of repeated keys) must not fail it; the rest must."""
    rng = np.random.default_rng(5)
    k, n = rng.permutation(3000) // (2 if "repeated" in keys else 1), 30_000
    k = k * (1 if keys in ("dense", "repeated") else 10 ** 5)
    t = L if keys == "wide" else I
    plan = _plan(k, k[rng.integers(0, 3000, n)], t, t, bpay=[(L, np.arange(3000), None)], ppay=[(F, rng.random(n), None)])
    want, rp = run_oracle(plan), _resident(plan, gpu_ctx)
    done_without, failed = [], []
    gpu_ctx.set_option(_lib.CJ_OPT_BUFFER_CACHE_BYTES, 0)
    try:
        used0, _ = gpu_ctx.memory()
        for at in range(1, 60):
            gpu_ctx.set_option(_lib.CJ_OPT_FAIL_ALLOC_AT, at)
            try:
                got, _ = run_product(rp, gpu_ctx, _lib.CJ_EXEC_RESULT_ON_DEVICE)
                reached = gpu_ctx.get_option(_lib.CJ_OPT_FAIL_ALLOC_AT) == 0
                assert_same(got, want, f"{keys}, allocation {at}")
                if not reached:
                    break
                done_without.append(at)
            except CJError as e:
                assert e.status == 4 and "injected" in str(e)
                failed.append(at)
            gpu_ctx.set_option(_lib.CJ_OPT_FAIL_ALLOC_AT, 0)
            assert gpu_ctx.memory()[0] == used0
        assert not reached and len(failed) >= 2
        assert len(done_without) >= {"dense": 3, "spread": 3, "wide": 3, "repeated": 7, "repeated_spread": 8}[keys]
    finally:
        gpu_ctx.set_option(_lib.CJ_OPT_FAIL_ALLOC_AT, 0)
        gpu_ctx.set_option(_lib.CJ_OPT_BUFFER_CACHE_BYTES, 16 << 30)
        for t in rp.inputs:
            t.free()


def test_server_worker_keeps_to_the_estimate():
    """Two matches per probe row: a context by itself makes room for them at
    once, a server's worker, whose memory others share, when it has counted."""
    rng = np.random.default_rng(6)
    bkeys = rng.permutation(np.repeat(np.arange(4000), 2))
    pkeys = rng.integers(0, 4000, 50_000)
    plan = _plan(bkeys, pkeys, bpay=[(L, np.arange(8000), None)])
    srv = Server(slots=1)
    try:
        res, st = srv.wait(srv.submit(plan))
        got = oa.PagedResult.from_result(res)
        res.free()
    finally:
        srv.close()
    assert_same(got, run_oracle(plan))
    assert st["probe_reruns"] == 1


def test_batch_gives_match_arrays_back():
    """Eight joins of a chain over 8M rows: a level's match arrays (32 MB)
    are gathered through and given back. Decoded columns (9 x 33 MB), a row-id
    vector per level and the result stay: 620 MB, and 190 more if the levels'
    match arrays stayed too."""
    n, joins = 8_000_000, 8
    rng = np.random.default_rng(7)
    fk = encode_column(I, rng.integers(0, 1000, n).astype(np.int32))
    plan = Plan()
    plan.inputs = [ColumnarTable(n, [fk] * (joins + 1))]
    left = plan.new_scan_node(0, [(i, I) for i in range(joins + 1)])
    for k in range(joins):
        plan.inputs.append(ColumnarTable(1000, [encode_column(I, rng.permutation(1000).astype(np.int32))]))
        scan = plan.new_scan_node(k + 1, [(0, I)])
        last = k == joins - 1
        left = plan.new_join_node(True, left, scan, k, 0, [(joins, I)] if last else [(i, I) for i in range(joins + 1)])
    plan.root = left
    ctx = Context(0)
    ctx.set_option(_lib.CJ_OPT_BUFFER_CACHE_BYTES, 0)
    rp = _resident(plan, ctx)
    try:
        before = ctx.memory()[1]
        res, sts, _ = execute_batch([rp], ctx, _lib.CJ_EXEC_RESULT_ON_DEVICE)
        grown = ctx.memory()[1] - before  # the pool keeps what it has reserved
        assert sts == [0] and res[0].num_rows == n
        res[0].free()
        assert grown < 720 << 20
    finally:
        for t in rp.inputs:
            t.free()
        ctx.close()
