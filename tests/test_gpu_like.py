"""GPU: LIKE over short strings against the oracle where groups of four
characters are skipped: every distance of a match, a near match, a newline,
a multi-byte character and a byte that is no UTF-8 from a '%' and from the
string's end."""
import numpy as np
import pytest

from calamarijoins_b200 import ColumnarTable, Comparison, DataType, LogicalOperation, encode_column
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


@pytest.mark.parametrize("rows", [1, 31, 33, 2047, 2048, 2049, 5000])
@pytest.mark.parametrize("keep", [0, 1, 50, 100])
def test_text_beside_other_conditions(gpu_ctx, rows, keep):
    """Text is compared for the rows that the other side of an AND leaves,
    around the 2,048 rows of a block: any order and nesting, under NOT and OR."""
    rng = np.random.default_rng(rows + keep)
    texts = [None if rng.random() < 0.1 else "ab"[int(rng.integers(2))] * int(rng.integers(0, 9)) for _ in range(rows)]
    texts = [t if t is None else (t * (2000 if rng.random() < 0.002 else 1)).encode() for t in texts]
    t = ColumnarTable(rows, [encode_column(DataType.INT32, rng.integers(0, 100, rows).astype(np.int32)),
                             encode_column(DataType.VARCHAR, texts)])
    A, O, N = LogicalOperation.makeAnd, LogicalOperation.makeOr, LogicalOperation.makeNot
    num, like, eq = Comparison(0, Comparison.LT, keep), Comparison(1, Comparison.LIKE, "%bb%"), Comparison(1, Comparison.GEQ, "ab")
    for pred in (A(num, like), A(like, num), A(A(eq, num), N(like)), N(A(num, N(like))), O(A(num, like), eq),
                 A(O(like, num), N(O(eq, like))), A(num, A(Comparison(1, Comparison.IS_NOT_NULL), N(N(like))))):
        want, sel = oa.oracle_filter(t, pred, [0, 1])
        got = gpu_filter(gpu_ctx, t, pred, [0, 1])
        assert got.num_rows == int(sel.sum())
        assert_same(got, want)


@pytest.mark.parametrize("rows", [302_000, 610_001, 1_215_003])
def test_rows_per_block(gpu_ctx, rows):
    """Tables whose blocks take 256, 512 and 1,024 rows at a time."""
    rng = np.random.default_rng(rows)
    words = [b"", b"a", b"qz", b"aqzb", b"xxqyzz", b"a\nqz"]
    texts = [words[k] for k in rng.integers(0, len(words), rows)]
    t = ColumnarTable(rows, [encode_column(DataType.INT32, np.arange(rows, dtype=np.int32)),
                             encode_column(DataType.VARCHAR, texts, (rng.random(rows) >= 0.1).astype(np.uint8))])
    like = Comparison(1, Comparison.LIKE, "%_qz%")
    for pred in (like, LogicalOperation.makeAnd(like, Comparison(0, Comparison.LT, rows // 3))):
        want, sel = oa.oracle_filter(t, pred, [0])
        got = gpu_filter(gpu_ctx, t, pred, [0])
        assert got.num_rows == int(sel.sum())
        assert_same(got, want)
