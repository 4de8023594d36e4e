"""GPU: joins over unique build keys (k_unique.cu) against the oracle: the
probe that reads the key column's pages and writes the result's, at the
edges of its pages and steps, and every kind of table at the edges of the
key range."""
import numpy as np
import pytest

from calamarijoins_b200 import ColumnarTable, DataType, Plan, ResidentTable, _lib, encode_column
from tests.helpers import assert_same, run_oracle, run_product

pytestmark = pytest.mark.gpu
I, L, F, V = DataType.INT32, DataType.INT64, DataType.FP64, DataType.VARCHAR
LO, HI = -(2 ** 31) + 1, 2 ** 31 - 1  # INT32_MIN is the intermediates' NULL
NP = {I: np.int32, L: np.int64, F: np.float64}


def _plan(bkeys, pkeys, bt=I, pt=I, bvalid=None, pvalid=None, bpay=(), ppay=(), out=None):
    """Tables of a key and payload columns (type, values, valid); output every column, or `out`."""
    plan = Plan()
    types = [bt] + [t for t, _, _ in bpay], [pt] + [t for t, _, _ in ppay]
    cols = [[encode_column(bt, bkeys.astype(NP[bt]), bvalid)], [encode_column(pt, pkeys.astype(NP[pt]), pvalid)]]
    for side, pay in enumerate((bpay, ppay)):
        cols[side] += [encode_column(t, v, ok) for t, v, ok in pay]
    plan.inputs = [ColumnarTable(len(bkeys), cols[0]), ColumnarTable(len(pkeys), cols[1])]
    plan.new_scan_node(0, list(enumerate(types[0])))
    plan.new_scan_node(1, list(enumerate(types[1])))
    allt = types[0] + types[1]
    plan.root = plan.new_join_node(True, 0, 1, 0, 0, [(i, allt[i]) for i in (out or range(len(allt)))])
    return plan


def _check(plan, ctx, kind):
    want = run_oracle(plan)
    rp = Plan()
    rp.nodes, rp.root = plan.nodes, plan.root
    rp.inputs = [ResidentTable(ctx, t) for t in plan.inputs]
    try:
        for p, flags in ((rp, _lib.CJ_EXEC_RESULT_ON_DEVICE), (rp, 0), (plan, 0)):
            got, st = run_product(p, ctx, flags)
            assert_same(got, want, kind)
            assert (st.exec["num_direct_joins"], st.exec["num_open_joins"]) == \
                {"direct": (1, 0), "open": (0, 1), "hash": (0, 0)}[kind]
    finally:
        for t in rp.inputs:
            t.free()


@pytest.mark.parametrize("null", [0.0, 0.02, 0.5, 0.97, 1.0])
@pytest.mark.parametrize("rows", [65, 1984, 1985, 2048, 2049, 70_001])
@pytest.mark.parametrize("gap", [1, 1000])
def test_key_pages(gpu_ctx, rows, null, gap):
    """NULL shares from none to all: dense pages, pages of about 2,020 rows,
    pages of more rows than a step takes (up to 65,504), pages without a
    value."""
    rng = np.random.default_rng(rows + int(100 * null))
    nb = min(rows, 3000)
    bkeys = rng.permutation(nb) * gap
    pkeys = bkeys[rng.integers(0, nb, rows)] + gap * nb * (rng.random(rows) < 0.2)
    ok = (rng.random(rows) >= null).astype(np.uint8)
    plan = _plan(bkeys, pkeys, pvalid=ok, bpay=[(L, rng.integers(0, 1 << 60, nb), None)],
                 ppay=[(F, rng.random(rows), None), (I, np.arange(rows), None)])
    _check(plan, gpu_ctx, "direct" if gap == 1 else "open")


@pytest.mark.parametrize("nb", [65, 1000, 8192, 8193, 40_000])
@pytest.mark.parametrize("bt,pt", [(I, I), (L, L), (I, L), (L, I)])
def test_key_types_and_range_edges(gpu_ctx, nb, bt, pt):
    """Direct-mapped ranges at both ends of INT32 and, for INT64 build keys,
    across and beyond them; probe keys around, below and far above."""
    rng = np.random.default_rng(nb)
    starts = [LO, HI - nb + 1, -nb // 2]
    if bt == L:
        starts += [HI - nb // 2, -(2 ** 31) - nb // 2, 2 ** 40, -(2 ** 62)]
    for lo in starts:
        bkeys = lo + rng.permutation(nb).astype(object)
        pkeys = np.array([lo + int(x) for x in rng.integers(-nb, 2 * nb, 5000 + 2 * nb)] + [LO, HI, 0, lo, lo + nb - 1], object)
        if pt == I:
            pkeys = np.clip(pkeys, LO, HI)
        else:
            pkeys[:50] += 2 ** 32  # equal to build keys in their low 32 bits
        plan = _plan(np.array(bkeys), pkeys, bt, pt, bpay=[(I, rng.integers(0, 100, nb), None)])
        _check(plan, gpu_ctx, "direct")


@pytest.mark.parametrize("pt", [I, L])
def test_open_range_edges(gpu_ctx, pt):
    """Spread INT32 keys that span all of INT32, with probe keys next to
    each, and INT64 probe keys that share their low 32 bits."""
    rng = np.random.default_rng(9)
    bkeys = np.unique(np.concatenate([[LO, LO + 2, HI - 2, HI], rng.integers(LO, HI, 20_000)]))
    rng.shuffle(bkeys)
    pkeys = np.concatenate([bkeys, bkeys + 1, bkeys - 1, [LO, HI]])
    pkeys = np.clip(pkeys, LO, HI) if pt == I else np.concatenate([pkeys, bkeys + 2 ** 32, bkeys - 2 ** 33])
    plan = _plan(bkeys, pkeys, I, pt, bpay=[(L, rng.integers(0, 1 << 60, len(bkeys)), None)])
    _check(plan, gpu_ctx, "open")


@pytest.mark.parametrize("gap", [1, 777])
@pytest.mark.parametrize("cols", ["nulls", "mixed", "many", "text"])
def test_result_columns(gpu_ctx, cols, gap):
    """Columns that the probe writes beside columns with NULLs (written
    through row ids), more columns than it takes (8), and VARCHARs."""
    rng = np.random.default_rng(4)
    nb, n = 9000, 30_000
    bkeys = rng.permutation(nb) * gap
    pkeys = bkeys[rng.integers(0, nb, n)] + gap * nb * (rng.random(n) < 0.3)

    def pay(t, rows, null):
        ok = (rng.random(rows) >= 0.2).astype(np.uint8) if null else None
        if t == V:
            return (V, ["x" * int(k) for k in rng.integers(0, 40, rows)], ok)
        return (t, rng.integers(0, 10 ** 6, rows), ok)

    which = {"nulls": [(I, 1), (L, 1), (F, 1)], "mixed": [(I, 0), (L, 1), (F, 0)],
             "many": [(t, k % 2) for k, t in enumerate([I, L, F] * 3)], "text": [(V, 1), (I, 0), (L, 1)]}[cols]
    plan = _plan(bkeys, pkeys, bpay=[pay(t, nb, x) for t, x in which], ppay=[pay(t, n, x) for t, x in which])
    _check(plan, gpu_ctx, "direct" if gap == 1 else "open")


@pytest.mark.parametrize("case", ["one_repeat", "all_equal", "repeat_spread"])
def test_repeated_keys_go_on(gpu_ctx, case):
    rng = np.random.default_rng(3)
    nb, n = 9000, 20_000
    bkeys = rng.permutation(nb) * (1000 if case == "repeat_spread" else 1)
    if case == "all_equal":
        bkeys = np.full(nb, 5)
        n = nb + 1
    else:
        bkeys[17] = bkeys[4000]
    pkeys = bkeys[rng.integers(0, nb, n)] + (rng.random(n) < 0.99 if case == "all_equal" else 0)
    _check(_plan(bkeys, pkeys, bpay=[(L, rng.integers(0, 1 << 60, nb), None)]), gpu_ctx, "hash")


def test_joins_in_a_row(gpu_ctx):
    """A chain whose joins use every kind of table, so that each counts its
    matches from zero: a nested loop, a repeated key, direct, open, direct."""
    rng = np.random.default_rng(8)
    n = 50_000
    sizes, plan = [20, 500, 3000, 4000, 9000], Plan()
    dims = [rng.permutation(s) for s in sizes]
    dims[1][3] = dims[1][9]
    dims[3] = dims[3] * 5000
    plan.inputs = [ColumnarTable(n, [encode_column(I, d[rng.integers(0, len(d), n)].astype(np.int32)) for d in dims])]
    left = plan.new_scan_node(0, [(i, I) for i in range(5)])
    types = [I] * 5
    for k, d in enumerate(dims):
        plan.inputs.append(ColumnarTable(len(d), [encode_column(I, d.astype(np.int32)),
                                                  encode_column(I, np.arange(len(d), dtype=np.int32))]))
        scan = plan.new_scan_node(k + 1, [(0, I), (1, I)])
        left = plan.new_join_node(True, left, scan, k, 0, list(enumerate(types)) + [(len(types) + 1, I)])
        types = types + [I]
    plan.root = left
    want = run_oracle(plan)
    for flags in (0, _lib.CJ_EXEC_RESULT_ON_DEVICE):
        got, _ = run_product(plan, gpu_ctx, flags)
        assert_same(got, want)


def _multi_case(case, rng):
    nb = 20_000
    if case == "twice":
        k = np.concatenate([np.arange(nb // 2)] * 2)
    elif case == "heavy":  # runs of 1, 32, 33, 300 and 5,000 rows
        k = np.concatenate([np.arange(nb - 5365), np.full(32, 7), np.full(33, 8), np.full(300, 9), np.full(5000, 10)])
    elif case == "sparse":  # one repeat over a range of 3.9 values per row
        k = rng.choice(int(3.9 * nb), nb, replace=False)
        k[5] = k[6]
    elif case == "edge":  # at the top of INT32
        k = HI - rng.integers(0, nb // 2, nb)
    else:  # all rows one key
        k = np.full(3000, 42)
    return rng.permutation(k)


@pytest.mark.parametrize("case", ["twice", "heavy", "sparse", "edge", "one_key"])
@pytest.mark.parametrize("bt,pt", [(I, I), (L, I), (I, L)])
def test_repeated_dense_keys(gpu_ctx, case, bt, pt):
    """The table of repeated dense keys: keys of one row, a few and many
    (above and below a warp's rounds), NULLs on both sides, results larger
    than the room made for them, payloads written by the probe and through
    row ids."""
    rng = np.random.default_rng(len(case))
    bkeys = _multi_case(case, rng)
    nb, n = len(bkeys), 25_000
    pkeys = np.clip(bkeys[rng.integers(0, nb, n)] + rng.integers(0, 2, n) * rng.integers(0, nb, n), LO, HI)
    if case == "heavy":
        pkeys[rng.random(n) < 0.9] = 100  # keep the 5,000-row key rare
    if case == "one_key":
        pkeys[100:] = 41
    bok = (rng.random(nb) >= 0.05).astype(np.uint8)
    pok = (rng.random(n) >= 0.05).astype(np.uint8)
    plan = _plan(bkeys, pkeys, bt, pt, bok, pok,
                 bpay=[(L, np.arange(nb), None), (I, rng.integers(0, 99, nb), (rng.random(nb) > 0.5).astype(np.uint8))],
                 ppay=[(F, rng.random(n), None)])
    _check(plan, gpu_ctx, "hash")


def test_repeated_dense_keys_in_a_chain(gpu_ctx):
    """Repeated keys below the root: row ids only, and rows of an
    intermediate as the probe side."""
    rng = np.random.default_rng(6)
    n, d = 30_000, [np.concatenate([rng.permutation(400)] * 3), np.concatenate([rng.permutation(900)] * 2)]
    plan = Plan()
    plan.inputs = [ColumnarTable(n, [encode_column(I, x[rng.integers(0, len(x), n)].astype(np.int32),
                                                   (rng.random(n) > 0.1).astype(np.uint8)) for x in d])]
    left = plan.new_scan_node(0, [(0, I), (1, I)])
    types = [I, I]
    for k, x in enumerate(d):
        plan.inputs.append(ColumnarTable(len(x), [encode_column(I, x.astype(np.int32)),
                                                  encode_column(L, np.arange(len(x)))]))
        scan = plan.new_scan_node(k + 1, [(0, I), (1, L)])
        left = plan.new_join_node(True, left, scan, k, 0, list(enumerate(types)) + [(len(types) + 1, L)])
        types = types + [L]
    plan.root = left
    want = run_oracle(plan)
    for flags in (0, _lib.CJ_EXEC_RESULT_ON_DEVICE):
        got, _ = run_product(plan, gpu_ctx, flags)
        assert_same(got, want)


@pytest.mark.parametrize("nb", [65, 1000, 8193, 40_000])
@pytest.mark.parametrize("case", ["random", "top", "bottom", "whole", "repeat", "minus_one"])
@pytest.mark.parametrize("pt", [I, L])
def test_wide_open_addressing(gpu_ctx, nb, case, pt):
    """Spread INT64 keys: 16-byte slots whose empty key lies next to the
    keys' range, which may end at either end of INT64 (at both: the hash
    table), hold -1 and the slots' fill pattern, or repeat."""
    rng = np.random.default_rng(nb)
    bkeys = np.unique(rng.integers(-(2 ** 62), 2 ** 62, nb))
    bkeys[0], bkeys[-1] = -(2 ** 62) - 5, 2 ** 62 + 5
    if case in ("top", "whole"):
        bkeys[-1] = 2 ** 63 - 1
    if case in ("bottom", "whole"):
        bkeys[0] = -(2 ** 63)
    if case == "minus_one":
        bkeys[1:4] = [-1, 0, 5]
    if case == "repeat":
        bkeys[7] = bkeys[9]
    if pt == I:
        bkeys[4:40] = np.arange(36) * 1000 - 7000
    bkeys = rng.permutation(bkeys)
    n = 2 * nb + 5000
    pkeys = bkeys[rng.integers(0, len(bkeys), n)].copy()
    miss = rng.random(n) < 0.3
    pkeys[miss] ^= 1 << 20
    if pt == I:
        pkeys = np.where(rng.random(n) < 0.5, rng.integers(-20, 60, n) * 500, np.clip(pkeys, LO, HI))
    plan = _plan(bkeys, pkeys, L, pt, (rng.random(len(bkeys)) > 0.02).astype(np.uint8),
                 (rng.random(n) > 0.02).astype(np.uint8), bpay=[(I, np.arange(len(bkeys)), None)],
                 ppay=[(F, rng.random(n), None)])
    _check(plan, gpu_ctx, "hash")
