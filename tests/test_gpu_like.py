"""GPU: LIKE over short strings against the oracle where groups of four
characters are skipped: every distance of a match, a near match, a newline,
a multi-byte character and a byte that is no UTF-8 from a '%' and from the
string's end."""
import numpy as np
import pytest

from calamarijoins_b200 import ColumnarTable, Comparison, DataType, encode_column
from oracle import oracle_api as oa
from tests.helpers import assert_same
from tests.test_gpu_filter import gpu_filter

pytestmark = pytest.mark.gpu
SPECIAL = [b"q", b"qz", b"qq", b"\n", "é".encode(), "中".encode(), b"\xff", b"\xe4", b"\xc3", b""]


@pytest.mark.parametrize("pattern", ["%qz%", "%qz", "q%z", "%q_%", "%", "_%", "%é%", "%中", "a%", "%q%z%", "", "%%qz",
                                     "%_qz%", "aaaa%aaaa", "%aaaaaaaa"])
def test_like_skips(gpu_ctx, pattern):
    rng = np.random.default_rng(1)
    rows = []
    for n in range(0, 20):
        for at in range(n + 1):
            for s in SPECIAL:
                rows.append(b"a" * at + s + b"a" * (n - at))
                rows.append(b"a" * at + s + b"aqza" + SPECIAL[int(rng.integers(len(SPECIAL)))] + b"b" * (n - at))
    rows = [rows[i] for i in rng.permutation(len(rows))]
    t = ColumnarTable(len(rows), [encode_column(DataType.VARCHAR, rows)])
    for op in (Comparison.LIKE, Comparison.NOT_LIKE):
        pred = Comparison(0, op, pattern)
        want, sel = oa.oracle_filter(t, pred, [0])
        got = gpu_filter(gpu_ctx, t, pred, [0])
        assert got.num_rows == int(sel.sum()), pattern
        assert_same(got, want, pattern)
