"""GPU: which table serves a join, by the kernels that ran, against the
oracle: one case per rule of the choice and per fallback, so that a table that
is never built cannot pass for one that is."""
import numpy as np
import pytest

from calamarijoins_b200 import ColumnarTable, DataType, Plan, ResidentTable, _lib, encode_column
from tests.helpers import assert_same, run_oracle, run_product
from tests.test_gpu_unique import _plan

pytestmark = pytest.mark.gpu
I, L, F, V = DataType.INT32, DataType.INT64, DataType.FP64, DataType.VARCHAR
PROBES = {"probe_unique", "probe_multi", "probe_open_multi", "probe_hash", "nl_probe"}
PILED = np.arange(1, 2001, dtype=np.int64)
PILED = (PILED << 32) | ((PILED * 0x2545F491) & 0xFFFFFFFF)  # one hash for all
WHOLE = np.concatenate([[-(2 ** 63), 2 ** 63 - 1], np.arange(2000) * 10 ** 15])
SEQ = np.arange(3000)
SLOT32, SLOT64 = 10 ** 5, 10 ** 12


def _probes(plan, ctx, flags):
    ctx.set_option(_lib.CJ_OPT_PROFILE_KERNELS, 1)
    ctx.profile_reset()
    try:
        got, st = run_product(plan, ctx, flags)
        return got, st, PROBES & set(ctx.profile())
    finally:
        ctx.set_option(_lib.CJ_OPT_PROFILE_KERNELS, 0)


# build keys, their type, probe rows per build row, the kernels that probe
CASES = {
    "nested_loop": (SEQ[:64], I, 100, {"nl_probe"}),
    "dense": (SEQ, I, 5, {"probe_unique"}),
    "dense64": (SEQ + 2 ** 40, L, 5, {"probe_unique"}),
    "spread": (SEQ * SLOT32, I, 5, {"probe_unique"}),
    "spread64": (SEQ * SLOT64, L, 5, {"probe_unique"}),
    "whole": (WHOLE, L, 5, {"probe_unique", "probe_hash"}),
    "piled_up": (PILED, L, 5, {"probe_unique", "probe_hash"}),
    "dense_repeats": (SEQ // 2, I, 5, {"probe_unique", "probe_multi"}),
    "dense_repeats64": (SEQ // 2 - 2 ** 40, L, 1, {"probe_unique", "probe_multi"}),
    "four_values_a_row": (np.concatenate([SEQ * 4, [0]]), I, 1, {"probe_unique", "probe_multi"}),
    "five_values_a_row": (np.concatenate([SEQ * 5, [0]]), I, 5, {"probe_unique", "probe_open_multi"}),
    "spread_repeats": (SEQ // 2 * SLOT32, I, 5, {"probe_unique", "probe_open_multi"}),
    "spread_eight": (SEQ // 8 * SLOT32, I, 5, {"probe_unique", "probe_open_multi"}),
    "spread_repeats64": (SEQ // 2 * SLOT64, L, 4, {"probe_unique", "probe_open_multi"}),
    "few_probe_rows": (SEQ // 2 * SLOT64, L, 3.99, {"probe_unique", "probe_hash"}),
    "whole_repeats": (np.concatenate([WHOLE, WHOLE]), L, 5, {"probe_unique", "probe_hash"}),
    "piled_up_repeats": (np.concatenate([PILED, PILED[:50]]), L, 5, {"probe_unique", "probe_hash"}),
}


# from 4M probe rows on the number of keys decides, from 1M where there are
# fewer than four per build row: build keys, their type, the kernels that probe
MANY = 1 << 22
WIDE = np.arange(60_000)
PILED_WIDE = np.arange(1, 20_001, dtype=np.int64)
PILED_WIDE = (PILED_WIDE << 32) | ((PILED_WIDE * 0x2545F491) & 0xFFFFFFFF)
SAMPLED = {
    "hardly": (np.concatenate([WIDE, WIDE[:100]]) * 30_000, I, {"probe_unique", "probe_hash"}),
    "two": (WIDE // 2 * 30_000, I, {"probe_unique", "probe_hash"}),
    "two64": (WIDE // 2 * SLOT64, L, {"probe_unique", "probe_hash"}),
    "three": (WIDE // 3 * 30_000, I, {"probe_unique", "probe_open_multi"}),
    "three64": (WIDE // 3 * SLOT64, L, {"probe_unique", "probe_open_multi"}),
    "sampled64": (np.arange(700_000) // 3 * SLOT64, L, {"probe_unique", "probe_open_multi"}),
    "sampled_two": (np.arange(700_000) // 2 * 3000, I, {"probe_unique", "probe_hash"}),
    "piled_up_four": (np.repeat(PILED_WIDE, 4), L, {"probe_unique", "probe_open_multi", "probe_hash"}),
    "few_two": (np.arange(700_000) // 2 * 3000, I, {"probe_unique", "probe_hash"}),
    "few_three64": (np.arange(700_000) // 3 * SLOT64, L, {"probe_unique", "probe_open_multi"}),
    "whole_three": (np.repeat(WHOLE, 3), L, {"probe_unique", "probe_hash"}),
}


@pytest.mark.parametrize("case", list(SAMPLED))
def test_route_by_number_of_keys(gpu_ctx, case):
    """Every probe row matches: one run, with room for the mean number."""
    bkeys, kt, probes = SAMPLED[case]
    rng = np.random.default_rng(1)
    bkeys = rng.permutation(bkeys)
    n = MANY // 4 if "few" in case else MANY
    pkeys = bkeys[rng.integers(0, len(bkeys), n)]
    if "piled" in case or "sampled" in case:
        pkeys[rng.random(n) < 0.9] = bkeys.min() - 1
    plan = _plan(bkeys, pkeys, kt, kt, bpay=[(I, np.arange(len(bkeys)), None)])
    want = run_oracle(plan)
    rp = Plan()
    rp.nodes, rp.root = plan.nodes, plan.root
    rp.inputs = [ResidentTable(gpu_ctx, t) for t in plan.inputs]
    try:
        got, st, ran = _probes(rp, gpu_ctx, _lib.CJ_EXEC_RESULT_ON_DEVICE)
    finally:
        for t in rp.inputs:
            t.free()
    assert_same(got, want, case)
    assert ran == probes
    assert st.exec["probe_reruns"] == 0


@pytest.mark.parametrize("flags", [0, _lib.CJ_EXEC_RESULT_ON_DEVICE])
@pytest.mark.parametrize("case", list(CASES))
def test_route(gpu_ctx, case, flags):
    bkeys, kt, times, probes = CASES[case]
    rng = np.random.default_rng(1)
    n = int(len(bkeys) * times)
    bkeys = rng.permutation(bkeys)
    plan = _plan(bkeys, bkeys[rng.integers(0, len(bkeys), n)], kt, kt, bpay=[(L, np.arange(len(bkeys)), None)],
                 ppay=[(F, rng.random(n), None)])
    want = run_oracle(plan)
    rp = Plan()
    rp.nodes, rp.root = plan.nodes, plan.root
    rp.inputs = [ResidentTable(gpu_ctx, t) for t in plan.inputs]
    try:
        got, st, ran = _probes(rp, gpu_ctx, flags)
    finally:
        for t in rp.inputs:
            t.free()
    assert_same(got, want, case)
    assert ran == probes
    assert (st.exec["num_direct_joins"], st.exec["num_open_joins"]) == \
        {"dense": (1, 0), "dense64": (1, 0), "spread": (0, 1)}.get(case, (0, 0))


def test_no_dense_keys_option(gpu_ctx):
    """CJ_OPT_DENSE_KEYS = 0: the hash table for every join."""
    rng = np.random.default_rng(2)
    was = gpu_ctx.get_option(_lib.CJ_OPT_DENSE_KEYS)
    plan = _plan(rng.permutation(SEQ), rng.integers(0, 3000, 9000), bpay=[(L, SEQ, None)])
    gpu_ctx.set_option(_lib.CJ_OPT_DENSE_KEYS, 0)
    try:
        got, _, ran = _probes(plan, gpu_ctx, 0)
    finally:
        gpu_ctx.set_option(_lib.CJ_OPT_DENSE_KEYS, was)
    assert_same(got, run_oracle(plan))
    assert ran == {"probe_hash"}


@pytest.mark.parametrize("empty", [False, True])
@pytest.mark.parametrize("ncols", [63, 64, 66, 90])
def test_many_small_host_columns(gpu_ctx, ncols, empty):
    """Host columns that go up in one copy, more of them than the status block
    tracks (64): a join whose payloads all lie beside its two keys."""
    rng = np.random.default_rng(ncols)
    n, half = 900, ncols // 2
    valid = (rng.random(n) > 0.2).astype(np.uint8)

    def cols(k):
        out = [encode_column(I, rng.permutation(n).astype(np.int32))]
        for c in range(k - 1):
            t, ok = (I, L, F, V)[c % 4], valid if c % 3 == 1 else None
            v = ["t%d" % x for x in rng.integers(0, 10 ** 5, n)] if t == V else rng.integers(0, 10 ** 6, n)
            out.append(encode_column(t, v, ok))
        return out

    left, right = cols(half), cols(ncols - half)
    if empty:
        right = [encode_column(c.type, [] if c.type == V else np.zeros(0)) for c in right]
    plan = Plan()
    plan.inputs = [ColumnarTable(n, left), ColumnarTable(0 if empty else n, right)]
    plan.new_scan_node(0, [(i, c.type) for i, c in enumerate(left)])
    plan.new_scan_node(1, [(i, c.type) for i, c in enumerate(right)])
    plan.root = plan.new_join_node(True, 0, 1, 0, 0, [(i, c.type) for i, c in enumerate(left + right)])
    for flags in (0, _lib.CJ_EXEC_RESULT_ON_DEVICE):
        got, _ = run_product(plan, gpu_ctx, flags)
        assert_same(got, run_oracle(plan), f"{ncols} columns")
        assert got.num_rows == (0 if empty else n)
