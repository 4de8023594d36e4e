"""GPU: probes of repeated keys with several matches a row, against the
oracle: matches per row on both sides of what the probe packs (3), of its
buffer (320) and of a warp, mixed in one page, by one block per step of the
probe side and by two, four and eight (few probe rows)."""
import numpy as np
import pytest

from calamarijoins_b200 import DataType
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
