"""GPU: joins over repeated build keys that are not dense (an open-addressing
table with a count per key, k_unique.cu), against the oracle: every number of
rows per key that the probe treats in its own way, every pair of key types,
NULLs, intermediates, and the keys that go on to the hash table."""
import numpy as np
import pytest

from calamarijoins_b200 import DataType
from tests.helpers import assert_same, run_oracle, run_product
from tests.test_gpu_unique import _check, _plan

pytestmark = pytest.mark.gpu
I, L, F, V = DataType.INT32, DataType.INT64, DataType.FP64, DataType.VARCHAR


def _keys(rng, distinct, bt):
    """Spread keys with both ends of the type's range but one value."""
    lo, hi = (-(2 ** 31) + 1, 2 ** 31 - 1) if bt == I else (-(2 ** 63), 2 ** 63 - 2)
    k = np.unique(np.concatenate([[lo, hi], rng.integers(lo, hi, distinct)]))
    rng.shuffle(k)
    return k


@pytest.mark.parametrize("per_key", [1, 2, 3, 4, 32, 33, 300])
@pytest.mark.parametrize("bt,pt", [(I, I), (L, L), (I, L), (L, I)])
def test_rows_per_key(gpu_ctx, bt, pt, per_key):
    """`per_key` rows for a fifth of the keys, one for the others (two keys
    repeat at least), 5 % NULL build keys; probe keys next to the build's."""
    rng = np.random.default_rng(per_key)
    k = _keys(rng, 3000 if per_key < 10 else 400, bt)
    bkeys = np.concatenate([np.repeat(k[:len(k) // 5], per_key), k[len(k) // 5:], k[:2]])
    rng.shuffle(bkeys)
    n = 4 * len(bkeys) + 2500  # a quarter of that, and the hash table serves it
    src = k if (bt, pt) != (L, I) else np.concatenate([k, rng.integers(-(2 ** 31) + 1, 2 ** 31, 50)])
    if (bt, pt) == (L, I):
        bkeys[:200] = rng.integers(-50, 50, 200)  # some that INT32 probe keys meet
        src = np.arange(-60, 60)
    pkeys = src[rng.integers(0, len(src), n)] + rng.integers(0, 2, n)
    if pt == I:
        pkeys = np.clip(pkeys, -(2 ** 31) + 1, 2 ** 31 - 1)
    bok, pok = (rng.random(len(bkeys)) >= 0.05).astype(np.uint8), (rng.random(n) >= 0.05).astype(np.uint8)
    plan = _plan(bkeys, pkeys, bt, pt, bvalid=bok, pvalid=pok, bpay=[(L, rng.integers(0, 1 << 60, len(bkeys)), None)],
                 ppay=[(F, rng.random(n), None)])
    _check(plan, gpu_ctx, "hash")


@pytest.mark.parametrize("cols", ["nulls", "text"])
def test_result_columns(gpu_ctx, cols):
    rng = np.random.default_rng(6)
    nb, n = 9000, 36_001
    bkeys = (rng.permutation(nb) // 2) * 777_777
    pkeys = bkeys[rng.integers(0, nb, n)] + (rng.random(n) < 0.3)
    ok = lambda rows: (rng.random(rows) >= 0.2).astype(np.uint8)
    pay = lambda rows: [(L, rng.integers(0, 1 << 60, rows), ok(rows)), (I, rng.integers(0, 99, rows), None)] + \
        ([(V, ["y" * int(k) for k in rng.integers(0, 30, rows)], ok(rows))] if cols == "text" else [])
    _check(_plan(bkeys, pkeys, L, L, bpay=pay(nb), ppay=pay(n)), gpu_ctx, "hash")


@pytest.mark.parametrize("case", ["whole", "piled_up", "piled_up_repeats", "wide_dense"])
def test_keys_that_go_on(gpu_ctx, case):
    """All of INT64's range (no key is free for empty slots), keys whose
    hashes are one (walks given up), and a range between dense and spread."""
    rng = np.random.default_rng(7)
    hi = np.arange(1, 2001, dtype=np.int64)
    if case == "whole":
        bkeys = np.concatenate([[-(2 ** 63), 2 ** 63 - 1], rng.integers(-(2 ** 62), 2 ** 62, 2000)])
        bkeys = np.concatenate([bkeys, bkeys[:900]])
    elif case == "wide_dense":
        bkeys = np.concatenate([np.arange(3000) * 6, np.arange(100) * 6])
    else:
        bkeys = (hi << 32) | ((hi * 0x2545F491) & 0xFFFFFFFF)
        if case == "piled_up_repeats":
            bkeys = np.concatenate([bkeys, bkeys[:50]])
    rng.shuffle(bkeys)
    pkeys = np.concatenate([bkeys[rng.integers(0, len(bkeys), 13_000)], bkeys + 1 if case != "whole" else bkeys])
    _check(_plan(bkeys, pkeys, L, L, bpay=[(I, rng.integers(0, 99, len(bkeys)), None)]), gpu_ctx, "hash")


def test_large_and_rerun(gpu_ctx):
    """More than a block's rows in every pass, and a result far above the
    room that the mean number of rows per key suggests."""
    rng = np.random.default_rng(11)
    k = np.unique(rng.integers(-(2 ** 62), 2 ** 62, 150_000))
    bkeys = np.concatenate([k, k[:60_000], np.repeat(k[:3], 40)])
    rng.shuffle(bkeys)
    pkeys = np.concatenate([k[rng.integers(0, len(k), 850_000)], np.repeat(k[0], 60_000), np.repeat(k[1], 3000)])
    rng.shuffle(pkeys)
    plan = _plan(bkeys, pkeys, L, L, bpay=[(L, np.arange(len(bkeys)), None)], ppay=[(I, np.arange(len(pkeys)), None)])
    want = run_oracle(plan)
    got, st = run_product(plan, gpu_ctx)
    assert_same(got, want, "rerun")
    assert st.exec["probe_reruns"] == 1
