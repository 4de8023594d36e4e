"""Cases for timing the framework through its public entry points.

A case is a dict of plain values. `listed()` names the standing ones, `draw(rng)` gives more of the same ranges,
`prepare(case, seed)` makes what a program holds before the call (tables and plans), `run(state)` is one call, and
`work(case)` is what the call cannot do without: every page of every column that the plan names read once, every
result page written once.

Kinds of case:

  join    two tables, one equi-join (`execute_raw`, or `execute` with pages in host memory)
  star    a left-deep chain of a fact table with several filtered dimensions, VARCHAR outputs (`execute_raw`)
  batch   many small chain plans in one call (`execute_batch`), or captured once and replayed (`PreparedBatch`)
  filter  a predicate over a resident table (`ResidentTable.filter`)

Tables are made on the GPU in the paged format, packed as the format's own writer packs them (a page takes rows while
they fit), and adopted by the library without a copy; host cases bring them to page-locked memory.

A join's rows come in no stated order, and two runs of one plan differ in it. `Rows` therefore reads a result column by
column with the rows sorted, when somebody asks for a column: the call itself is over by then, its pages are written.
Its arrays have room for `most_rows(case)` rows, whatever the seed, with zeros after the last.
"""
import ctypes
import math

import numpy as np
import torch

import calamarijoins_b200 as cj
from calamarijoins_b200 import DataType, _lib
from calamarijoins_b200.datagen import varchar_values
from calamarijoins_b200.predicate import Comparison, LogicalOperation

PAGE = cj.PAGE_SIZE
I32, I64, F64, STR = DataType.INT32, DataType.INT64, DataType.FP64, DataType.VARCHAR
TYPES = {"i32": I32, "i64": I64, "f64": F64, "str": STR}
WIDTH = {I32: 4, I64: 8, F64: 8}
FULL = {I32: 1984, I64: 1007, F64: 1007}  # rows of a full page without NULLs
INT32_MAX = 2 ** 31 - 1

JOIN = {"kind": "join", "build": 0, "probe": 0, "key": "i32", "gap": 1, "dup": 0.0, "zipf": 0.0, "outside": 0.0,
        "key_null": 0.0, "payload": "i32", "fact": "i32", "null": 0.0, "host": False}


def listed():
    return [
        # a lookup against a table of a few rows (the nested loop's range): all latency
        {**JOIN, "name": "join_tiny", "build": 50, "probe": 1000},
        # the drop-in call of a small query: pages in host memory, result in host memory
        {**JOIN, "name": "join_small_host", "build": 3001, "probe": 40009, "zipf": 0.8, "key_null": 0.05,
         "fact": "i64", "host": True},
        # the benchmark's C1: 100K x 1M, INT64 payload on the fact side, 5 % NULL keys
        {**JOIN, "name": "join_c1", "build": 100_000, "probe": 1_000_000, "zipf": 1.0, "key_null": 0.05,
         "fact": "i64"},
        # the benchmark's C2, the headline: 4M x 64M, ids 0 ... 4M - 1, 30 % of the foreign keys dangling
        {**JOIN, "name": "join_c2", "build": 4_000_000, "probe": 64_000_000, "zipf": 0.8, "outside": 0.3,
         "key_null": 0.02, "payload": "i64", "fact": "f64"},
        # C2 with its ids spread 500x (ids of a sharded or hashed sequence)
        {**JOIN, "name": "join_spread", "build": 4_000_000, "probe": 64_000_000, "gap": 500, "zipf": 0.8,
         "outside": 0.3, "key_null": 0.02, "payload": "i64", "fact": "f64"},
        # C2 with keys that repeat on the build side (many-to-many)
        {**JOIN, "name": "join_repeated", "build": 4_000_000, "probe": 64_000_000, "dup": 0.25, "zipf": 0.8,
         "outside": 0.3, "key_null": 0.02, "payload": "i64", "fact": "f64"},
        # 64-bit ids over the whole range, NULLs in the payloads, odd sizes
        {**JOIN, "name": "join_int64", "build": 300_007, "probe": 5_000_011, "key": "i64", "gap": 1 << 40,
         "zipf": 0.5, "outside": 0.1, "key_null": 0.01, "payload": "i64", "fact": "i32", "null": 0.1},
        # names and texts on both sides, some of them NULL
        {**JOIN, "name": "join_text", "build": 120_000, "probe": 2_000_003, "zipf": 0.8, "outside": 0.1,
         "payload": "str", "fact": "str", "null": 0.05},
        # the benchmark's C3 at a quarter: six tables, dimensions already filtered, VARCHAR outputs
        {"name": "star_c3", "kind": "star", "fact": 9_000_000, "dims": 5, "scale": 0.25, "null": 0.0},
        # the benchmark's C4: plans of 2 to 4 tables, in one call, and as a captured graph
        {"name": "batch_small", "kind": "batch", "plans": 48, "max_build": 100_000, "max_probe": 300_000,
         "graph": False},
        {"name": "batch_graph", "kind": "batch", "plans": 32, "max_build": 1_000_000, "max_probe": 4_000_000,
         "graph": True},
        # the scan before a join: a range, a comparison of doubles and a LIKE
        {"name": "filter_10m", "kind": "filter", "rows": 10_000_000, "keep": 0.3, "text": True, "null": 0.05},
    ]


def _spread(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["join"] * 7 + ["star", "batch", "filter"])
    if kind == "star":
        return {"kind": kind, "fact": _spread(rng, 100_000, 8_000_000), "dims": rng.randint(2, 5),
                "scale": round(rng.uniform(0.02, 0.25), 3), "null": rng.choice([0.0, 0.05])}
    if kind == "batch":
        return {"kind": kind, "plans": rng.randint(4, 40), "max_build": _spread(rng, 1000, 500_000),
                "max_probe": _spread(rng, 10_000, 2_000_000), "graph": rng.random() < 0.5}
    if kind == "filter":
        return {"kind": kind, "rows": _spread(rng, 10_000, 12_000_000), "keep": round(rng.uniform(0.02, 0.9), 3),
                "text": rng.random() < 0.5, "null": rng.choice([0.0, 0.05, 0.3])}
    host = rng.random() < 0.25
    text = rng.random() < 0.2
    probe = _spread(rng, 500, 1_500_000 if host else 3_000_000 if text else 40_000_000)
    build = min(_spread(rng, 10, 4_000_000), max(10, probe // 2))
    key = rng.choice(["i32", "i32", "i64"])
    gap = rng.choice([1, 1, 3, 500 if key == "i32" else 1 << 30])
    return {**JOIN, "build": build, "probe": probe, "key": key, "gap": gap, "dup": rng.choice([0.0, 0.0, 0.25, 0.5]),
            "zipf": round(rng.choice([0.0, rng.uniform(0.1, 1.2)]), 2), "outside": round(rng.uniform(0, 0.5), 2),
            "key_null": rng.choice([0.0, 0.02, 0.2]),
            "payload": "str" if text else rng.choice(["i32", "i64", "f64"]),
            "fact": rng.choice(["i32", "i64", "f64"]), "null": rng.choice([0.0, 0.0, 0.1]), "host": host}


# ---- values -------------------------------------------------------------------------------------------------------


class _Maker:
    """Seeded columns on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed) * 7919 + 17)
        self.np = np.random.default_rng(int(seed))

    def rand(self, n):
        return torch.rand(n, generator=self.g, device="cuda", dtype=torch.float64)

    def ints(self, lo, hi, n, dtype=torch.int64):
        return torch.randint(lo, hi, (n,), generator=self.g, device="cuda", dtype=dtype)

    def perm(self, n):
        return torch.randperm(n, generator=self.g, device="cuda")

    def valid(self, n, null):
        return None if null <= 0 else torch.rand(n, generator=self.g, device="cuda") >= null

    def zipf(self, n, s, size):
        """`size` places in [0, n), place k about as often as (k + 1)^-s."""
        if s == 0:
            return self.ints(0, n, size)
        u = self.rand(size)
        if abs(s - 1.0) < 1e-9:
            x = 0.5 * torch.exp(u * math.log((n + 0.5) / 0.5))
        else:
            a, b = 0.5 ** (1 - s), (n + 0.5) ** (1 - s)
            x = (a + u * (b - a)) ** (1.0 / (1 - s))
        return torch.clamp(torch.floor(x + 0.5).long(), 1, n) - 1

    def foreign(self, keys, n, s, outside, top):
        """Foreign keys: Zipf(s) over `keys`, a share `outside` of them above every key."""
        fk = keys[self.perm(len(keys))][self.zipf(len(keys), s, n)]
        if outside > 0:
            m = torch.rand(n, generator=self.g, device="cuda") < outside
            fk = torch.where(m, self.ints(int(keys.max()) + 1, top, n), fk)
        return fk

    def payload(self, t, n, null=0.0, long_share=0.0):
        """Pages of a payload column."""
        valid = self.valid(n, null)
        if t == I32:
            return fixed_pages(I32, self.ints(-INT32_MAX, INT32_MAX, n, torch.int32), valid)
        if t == I64:
            return fixed_pages(I64, self.ints(-(2 ** 62), 2 ** 62, n), valid)
        if t == F64:
            return fixed_pages(F64, torch.randn(n, generator=self.g, device="cuda", dtype=torch.float64) * 1e6, valid)
        if long_share:
            col = cj.encode_column(STR, varchar_values(n, self.np, long_frac=long_share),
                                   None if valid is None else valid.cpu().numpy())
            return torch.from_numpy(np.array(col.pages)).cuda()
        sigma = 0.6
        z = torch.randn(n, generator=self.g, device="cuda", dtype=torch.float64)
        lens = torch.clamp(torch.round(torch.exp(z * sigma + math.log(20.0) - sigma * sigma / 2)), 0, 200).long()
        return text_pages(lens, valid, self.g)


# ---- pages --------------------------------------------------------------------------------------------------------


def _page_starts(weight, limit):
    """First rows of the pages: a page takes rows while their weights sum to at most `limit`."""
    n = len(weight)
    sums = torch.cat([weight.new_zeros(1), torch.cumsum(weight, 0)])
    nxt = (torch.searchsorted(sums, sums[:-1] + limit, right=True) - 1).to(torch.int32).cpu().numpy()
    starts, a = [], 0
    while a < n:
        starts.append(a)
        a = int(nxt[a])
    return torch.tensor(starts + [n], device="cuda", dtype=torch.int64)


def _put_header(pages, rows, values):
    h = pages.view(torch.int16).view(len(pages), PAGE // 2)
    h[:, 0] = rows.to(torch.int16)
    h[:, 1] = values.to(torch.int16)


def _put_bitmap(pages, starts, page_of, in_page, valid):
    """Each page's bitmap: ceil(rows / 8) bytes at its end."""
    nbytes = (starts[1:] - starts[:-1] + 7) // 8
    ends = torch.cumsum(nbytes, 0)
    at = (ends - nbytes)[page_of] + in_page // 8
    bits = torch.zeros(int(ends[-1]), device="cuda", dtype=torch.int32)
    one = (1 << (in_page % 8)).to(torch.int32)
    bits.index_add_(0, at, one if valid is None else torch.where(valid, one, torch.zeros_like(one)))
    owner = torch.repeat_interleave(torch.arange(len(nbytes), device="cuda"), nbytes)
    place = torch.arange(len(bits), device="cuda") - (ends - nbytes)[owner]
    pages.view(-1)[owner * PAGE + PAGE - nbytes[owner] + place] = bits.to(torch.uint8)


def fixed_pages(t, values, valid=None):
    """Pages of a fixed-width column."""
    n, w, dtype = len(values), WIDTH[t], {I32: torch.int32, I64: torch.int64, F64: torch.float64}[t]
    values = values.to(dtype)
    if valid is None and n >= FULL[t]:  # whole pages at once, the last one by itself
        full, r = n // FULL[t], FULL[t]
        pages = torch.zeros((full, PAGE), device="cuda", dtype=torch.uint8)
        pages.view(dtype).view(full, PAGE // w)[:, 1:1 + r] = values[:full * r].view(full, r)
        rows = torch.full((full,), r, device="cuda", dtype=torch.int64)
        _put_header(pages, rows, rows)
        nb = (r + 7) // 8
        pages[:, PAGE - nb:] = 255
        if r % 8:
            pages[:, PAGE - 1] = (1 << (r % 8)) - 1
        return torch.cat([pages, fixed_pages(t, values[full * r:])]) if n > full * r else pages
    if n == 0:
        return torch.zeros((0, PAGE), device="cuda", dtype=torch.uint8)
    ok = torch.ones(n, device="cuda", dtype=torch.bool) if valid is None else valid
    starts = _page_starts(1 + 8 * w * ok.long(), 8 * (PAGE - w))
    count = starts[1:] - starts[:-1]
    page_of = torch.repeat_interleave(torch.arange(len(count), device="cuda"), count)
    in_page = torch.arange(n, device="cuda") - starts[page_of]
    sums = torch.cat([starts.new_zeros(1), torch.cumsum(ok.long(), 0)])
    pages = torch.zeros((len(count), PAGE), device="cuda", dtype=torch.uint8)
    k = (sums[:-1] - sums[starts[page_of]])[ok]
    pages.view(dtype).view(-1)[page_of[ok] * (PAGE // w) + 1 + k] = values[ok]
    _put_header(pages, count, sums[starts[1:]] - sums[starts[:-1]])
    _put_bitmap(pages, starts, page_of, in_page, ok)
    return pages


def text_pages(lens, valid, g):
    """Pages of a VARCHAR column of random letters, no string longer than a page."""
    n = len(lens)
    ok = torch.ones(n, device="cuda", dtype=torch.bool) if valid is None else valid
    lens = torch.where(ok, lens, torch.zeros_like(lens))
    starts = _page_starts(1 + 16 * ok.long() + 8 * lens, 8 * (PAGE - 4))
    count = starts[1:] - starts[:-1]
    page_of = torch.repeat_interleave(torch.arange(len(count), device="cuda"), count)
    in_page = torch.arange(n, device="cuda") - starts[page_of]
    vsum = torch.cat([starts.new_zeros(1), torch.cumsum(ok.long(), 0)])
    csum = torch.cat([starts.new_zeros(1), torch.cumsum(lens, 0)])
    values, chars = vsum[starts[1:]] - vsum[starts[:-1]], csum[starts[1:]] - csum[starts[:-1]]
    at = torch.arange(PAGE, device="cuda")
    letters = torch.randint(97, 123, (len(count), PAGE), generator=g, device="cuda", dtype=torch.uint8)
    inside = (at >= (4 + 2 * values)[:, None]) & (at < (4 + 2 * values + chars)[:, None])
    pages = torch.where(inside, letters, torch.zeros_like(letters))
    k = (vsum[:-1] - vsum[starts[page_of]])[ok]
    end = (csum[1:] - csum[starts[page_of]])[ok]
    pages.view(torch.int16).view(-1)[page_of[ok] * (PAGE // 2) + 2 + k] = end.to(torch.int16)
    _put_header(pages, count, values)
    _put_bitmap(pages, starts, page_of, in_page, ok)
    return pages


# ---- tables and plans ---------------------------------------------------------------------------------------------

_CTX = None


def context():
    """The program's one device context."""
    global _CTX
    if _CTX is None:
        _CTX = cj.build_context(0)
    return _CTX


def resident(rows, types, pages):
    """A resident table over pages that are in device memory already."""
    n = len(types)
    handle = ctypes.c_void_p()
    torch.cuda.synchronize()
    _lib.check(_lib.lib().cj_table_from_device(
        context().handle, rows, n, (ctypes.c_int32 * n)(*[int(t) for t in types]),
        (ctypes.c_uint64 * n)(*[len(p) for p in pages]), (ctypes.c_void_p * n)(*[p.data_ptr() for p in pages]),
        ctypes.byref(handle)))
    t = cj.ResidentTable.from_handle(context(), handle.value, rows, types)
    t.adopted = pages
    return t


def on_host(rows, types, pages):
    """The same table with its pages in page-locked host memory."""
    cols = []
    for t, p in zip(types, pages):
        buf = cj.PinnedBuffer(max(p.numel(), 1))
        arr = buf.array[:p.numel()].reshape(len(p), PAGE)
        arr[:] = p.cpu().numpy()
        cols.append(cj.Column(t, arr, buf))
    return cj.ColumnarTable(rows, cols)


def _build_keys(m, case):
    distinct = max(1, int(case["build"] * (1 - case["dup"])))
    if case["key"] == "i32":
        gap = max(1, min(case["gap"], (INT32_MAX - 1) // 2 // distinct))
    else:
        gap = case["gap"]
    keys = m.perm(distinct) * gap
    if gap > 3 and case["key"] == "i64":
        keys = keys + m.ints(0, gap, distinct)
    rows = keys[torch.arange(case["build"], device="cuda") % distinct]  # none more than once more than another
    return rows[m.perm(len(rows))], keys


def _join(case, seed):
    m = _Maker(seed)
    key, bt, ft = TYPES[case["key"]], TYPES[case["payload"]], TYPES[case["fact"]]
    rows, distinct = _build_keys(m, case)
    top = INT32_MAX if key == I32 else 2 ** 62
    fk = m.foreign(distinct, case["probe"], case["zipf"], case["outside"], top)
    ids = torch.arange(case["probe"], device="cuda", dtype=torch.int32)
    build = ([key, bt], [fixed_pages(key, rows), m.payload(bt, case["build"], case["null"])])
    probe = ([key, ft], [fixed_pages(key, fk, m.valid(case["probe"], case["key_null"])),
                         m.payload(ft, case["probe"], case["null"])])
    out = [(0, key), (1, bt), (2, key), (3, ft)]
    if STR in (bt, ft):  # a row id beside the texts
        probe[0].append(I32)
        probe[1].append(fixed_pages(I32, ids))
        out.append((4, I32))
    make = on_host if case["host"] else resident
    plan = cj.Plan()
    plan.inputs = [make(case["build"], *build), make(case["probe"], *probe)]
    plan.new_scan_node(0, list(enumerate(build[0])))
    plan.new_scan_node(1, list(enumerate(probe[0])))
    plan.root = plan.new_join_node(True, 0, 1, 0, 0, out)
    return plan


STAR_ROWS = (2_500, 130_000, 1_200_000, 2_500_000, 4_200_000)
STAR_KEEP = (0.40, 0.40, 0.30, 0.20, 0.10)
STAR_ZIPF = (0.5, 1.0, 1.2, 1.0, 0.5)


def _star_kept(case):
    return [max(1, int(max(8, int(n * case["scale"])) * k)) for n, k in zip(STAR_ROWS, STAR_KEEP)][:case["dims"]]


def _star(case, seed):
    m = _Maker(seed)
    n, nd = case["fact"], case["dims"]
    plan = cj.Plan()
    pages, dims = [], []
    for d, kept in enumerate(_star_kept(case)):
        size = max(8, int(STAR_ROWS[d] * case["scale"]))
        domain = m.perm(size)
        keys = domain[torch.sort(m.perm(size)[:kept]).values]
        pages.append(fixed_pages(I32, m.foreign(domain, n, STAR_ZIPF[d], 0.0, INT32_MAX)))
        dims.append((kept, [fixed_pages(I32, keys), m.payload(STR, kept, case["null"], 1e-4)]))
    types = [I32] * nd + [STR, I32]
    pages += [m.payload(STR, n, case["null"]), fixed_pages(I32, torch.arange(n, device="cuda"))]
    plan.inputs = [resident(n, types, pages)] + [resident(k, [I32, STR], p) for k, p in dims]
    left = plan.new_scan_node(0, list(enumerate(types)))
    scans = [plan.new_scan_node(1 + d, [(0, I32), (1, STR)]) for d in range(nd)]
    for d in range(nd):
        left = plan.new_join_node(False, left, scans[d], d, 0, list(enumerate(types)) + [(len(types) + 1, STR)])
        types = types + [STR]
    plan.root = left
    return plan


def _chain_shapes(case):
    """(probe rows, build sizes) of a batch's plans: the sizes are the batch's, only the values are the seed's."""
    r = np.random.default_rng(case["plans"] * 1_000_003 + case["max_probe"])
    out = []
    for _ in range(case["plans"]):
        probe = int(10 ** r.uniform(3, math.log10(case["max_probe"])))
        out.append((probe, [int(10 ** r.uniform(1, math.log10(case["max_build"]))) for _ in range(r.integers(1, 4))]))
    return out


def _chains(case, seed):
    m = _Maker(seed)
    plans = []
    for probe, builds in _chain_shapes(case):
        pages, dims = [], []
        for nb in builds:
            keys = m.perm(nb)
            s, out = float(m.np.uniform(0, 1.2)), float(m.np.uniform(0, 0.3))
            pages.append(fixed_pages(I32, m.foreign(keys, probe, s, out, INT32_MAX), m.valid(probe, 0.01)))
            dims.append((nb, [fixed_pages(I32, keys), fixed_pages(I32, m.ints(0, 1 << 30, nb))]))
        pages.append(fixed_pages(I32, m.ints(0, 1 << 30, probe)))
        types = [I32] * len(pages)
        plan = cj.Plan()
        plan.inputs = [resident(probe, types, pages)] + [resident(k, [I32, I32], p) for k, p in dims]
        left = plan.new_scan_node(0, list(enumerate(types)))
        scans = [plan.new_scan_node(1 + d, [(0, I32), (1, I32)]) for d in range(len(dims))]
        for d, scan in enumerate(scans):
            left = plan.new_join_node(True, left, scan, d, 0, list(enumerate(types)) + [(len(types) + 1, I32)])
            types = types + [I32]
        plan.root = left
        plans.append(plan)
    return plans


def _filter(case, seed):
    m = _Maker(seed)
    n = case["rows"]
    types = [I32, I32, F64, STR] if case["text"] else [I32, I32, F64]
    pages = [fixed_pages(I32, torch.arange(n, device="cuda")), fixed_pages(I32, m.ints(0, 1_000_000, n),
                                                                          m.valid(n, case["null"])),
             m.payload(F64, n, case["null"])]
    if case["text"]:
        pages.append(m.payload(STR, n, case["null"]))
    pred = LogicalOperation.makeAnd(Comparison(1, Comparison.LT, int(1_000_000 * case["keep"])),
                                    Comparison(2, Comparison.LT, 1e6))
    if case["text"]:
        pred = LogicalOperation.makeAnd(pred, LogicalOperation.makeNot(Comparison(3, Comparison.LIKE, "%qz%")))
    return {"table": resident(n, types, pages), "pred": pred, "types": types}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "filter":
        return {"case": case, **_filter(case, seed)}
    if kind == "batch":
        plans = _chains(case, seed)
        descs = [cj.PlanDescriptor(p) for p in plans]
        state = {"case": case, "plans": plans, "descs": descs}
        if case["graph"]:
            state["graph"] = cj.PreparedBatch(plans, context(), _lib.CJ_EXEC_RESULT_ON_DEVICE, descs=descs)
        return state
    plan = _star(case, seed) if kind == "star" else _join(case, seed)
    return {"case": case, "plan": plan, "desc": cj.PlanDescriptor(plan)}


def run(state):
    case = state["case"]
    if case["kind"] == "filter":
        return Rows(state["table"].filter(state["pred"]), False, state)
    if case["kind"] == "batch":
        if case["graph"]:
            return Batch(state["graph"].run()[0], state)
        return Batch(cj.execute_batch(state["plans"], context(), _lib.CJ_EXEC_RESULT_ON_DEVICE,
                                      descs=state["descs"])[0], state)
    if case.get("host"):
        return Rows(cj.execute(state["plan"], context()), True, state)
    return Rows(cj.execute_raw(state["plan"], context(), _lib.CJ_EXEC_RESULT_ON_DEVICE, state["desc"])[0], True, state)


# ---- results ------------------------------------------------------------------------------------------------------


class _DevicePages:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n, PAGE), "typestr": "|u1", "data": (ptr, False), "version": 3}


def _columns(result):
    """[(type, pages on the GPU)] of a result, a filtered table or a host table."""
    if isinstance(result, cj.ColumnarTable):
        return [(c.type, torch.from_numpy(c.pages).cuda()) for c in result.columns]
    out, ptr, n = [], ctypes.c_void_p(), ctypes.c_uint64()
    types = result.types if isinstance(result, cj.ResidentTable) else None
    for c in range(len(types) if types is not None else result.num_columns):
        if types is not None:
            _lib.check(_lib.lib().cj_table_column_pages(result.handle, c, ctypes.byref(ptr), ctypes.byref(n)))
            t, k = types[c], n.value
        else:
            t, k, _ = result.column_info(c)
            _lib.check(_lib.lib().cj_result_column_device(result.handle, c, ctypes.byref(ptr)))
        pages = torch.as_tensor(_DevicePages(ptr.value, k), device="cuda") if k else \
            torch.zeros((0, PAGE), device="cuda", dtype=torch.uint8)
        out.append((t, pages))
    return out


def _rows_of(pages, rows):
    """Per row: its page, its place in the page, whether it is non-NULL, and its value's place in the page."""
    page_of = torch.repeat_interleave(torch.arange(len(pages), device="cuda"), rows)
    first = torch.cumsum(rows, 0) - rows
    in_page = torch.arange(len(page_of), device="cuda") - first[page_of]
    byte = PAGE - (rows[page_of] + 7) // 8 + in_page // 8
    ok = (pages.view(-1)[page_of * PAGE + byte].long() >> (in_page % 8)) & 1
    sums = torch.cumsum(ok, 0) - ok
    place = sums - sums[first.clamp(max=max(len(sums) - 1, 0))][page_of] if len(sums) else sums
    return page_of, ok.bool(), place


def _fixed(t, pages):
    """(values, 0 where NULL; 1 where not NULL) of a fixed-width column; doubles as their bits."""
    head = pages.view(torch.int16).view(len(pages), PAGE // 2)[:, :2].long() & 0xFFFF
    page_of, ok, place = _rows_of(pages, head[:, 0])
    w, dtype = WIDTH[t], torch.int32 if t == I32 else torch.int64
    at = page_of * (PAGE // w) + 1 + torch.where(ok, place, torch.zeros_like(place))
    got = pages.view(-1).view(dtype)[at]
    return torch.where(ok, got, torch.zeros_like(got)), ok.to(torch.uint8)


def _text(pages):
    """(first character's place in `pages`, length, 1 where not NULL) per row; a string over several pages has its
    pages' count negated as its length."""
    head = pages.view(torch.int16).view(len(pages), PAGE // 2)[:, :2].long() & 0xFFFF
    long_first, long_more = head[:, 0] == 0xFFFF, head[:, 0] == 0xFFFE
    rows = torch.where(long_first, 1, torch.where(long_more, 0, head[:, 0]))
    page_of, ok, place = _rows_of(pages, rows)
    is_long = long_first[page_of]
    ends = pages.view(torch.int16).view(-1)
    base = page_of * (PAGE // 2) + 2
    short = ok & ~is_long
    k = torch.where(short, place, torch.zeros_like(place))
    end = ends[base + k].long() & 0xFFFF
    beg = torch.where(k > 0, ends[base + (k - 1).clamp(min=0)].long() & 0xFFFF, torch.zeros_like(end))
    first = page_of * PAGE + 4 + 2 * head[:, 1][page_of] + beg
    starts = torch.nonzero(long_first).view(-1)
    nxt = torch.cat([torch.nonzero(~long_more).view(-1), torch.tensor([len(pages)], device="cuda")])
    length = torch.where(short, end - beg, torch.zeros_like(end))
    if len(starts):
        after = nxt[torch.searchsorted(nxt, starts, right=True)]
        length[is_long] = -(after - starts)
        first[is_long] = starts * PAGE
    return first, length, (ok | is_long).to(torch.uint8)


def _gather_text(pages, first, length):
    """All strings' characters, one after another, and their lengths."""
    flat, host = pages.view(-1), {}
    for i in torch.nonzero(length < 0).view(-1).tolist():
        p, n = int(first[i]) // PAGE, -int(length[i])
        chunk = pages[p:p + n].cpu().numpy()
        host[i] = np.concatenate([c[4:4 + int(c[2]) + 256 * int(c[3])] for c in chunk])
    size = length.clamp(min=0)
    for i, c in host.items():
        size[i] = len(c)
    total = torch.cumsum(size, 0)
    owner = torch.repeat_interleave(torch.arange(len(size), device="cuda"), size)
    at = torch.arange(len(owner), device="cuda") - (total - size)[owner]
    chars = flat[(first[owner] + at).clamp(max=flat.numel() - 1)] if len(owner) else flat[:0].clone()
    for i, c in host.items():
        chars[int(total[i]) - len(c):int(total[i])] = torch.from_numpy(c).cuda()
    return chars, size


def _order(fixed):
    """The rows' order by the fixed-width columns."""
    order = None
    for v, ok in reversed(fixed):
        for x in (v, ok):
            if x is ok and bool(ok.all()):
                continue
            order = torch.argsort(x, stable=True) if order is None else order[torch.argsort(x[order], stable=True)]
    return order


def most_rows(case):
    """Rows that a result's arrays have room for: more than any seed gives."""
    if case["kind"] == "filter":
        return case["rows"]
    if case["kind"] == "batch":
        return sum(probe * (2 * len(builds) + 1) for probe, builds in _chain_shapes(case))
    if case["kind"] == "star":
        out = float(case["fact"])
        for keep in STAR_KEEP[:case["dims"]]:
            out *= keep
        return min(case["fact"], int(3 * out) + 1000)
    return case["probe"] * math.ceil(1 / (1 - case["dup"]))


def _room(x, n):
    """`x` in an array of `n` values, zeros after the last."""
    return torch.cat([x[:n], x.new_zeros(max(0, n - len(x)))])


class Rows(dict):
    """A result's columns by name, with the rows in the order of their values (`sort`) or as they stand. A column is
    read from the result's pages when it is asked for."""

    def __init__(self, result, sort, state):
        self.result, self.sort, self.state, self.seen = result, sort, state, {}
        self.most = most_rows(state["case"])
        types = self.result.types if isinstance(self.result, cj.ResidentTable) else \
            [c.type for c in self.result.columns] if isinstance(self.result, cj.ColumnarTable) else \
            [self.result.column_info(c)[0] for c in range(self.result.num_columns)]
        names = {"rows": None}
        for c, t in enumerate(types):
            names.update(dict.fromkeys(["c%d" % c, "c%d_valid" % c] + (["c%d_lens" % c] if t == STR else [])))
        super().__init__(names)

    def _column(self, c):
        if "columns" not in self.seen:
            self.seen["columns"] = _columns(self.result)
            if self.sort:
                self.seen["order"] = _order([_fixed(t, p) for t, p in self.seen["columns"] if t != STR])
        t, pages = self.seen["columns"][c]
        order = self.seen.get("order")
        got = _text(pages) if t == STR else _fixed(t, pages)
        if order is not None:
            got = tuple(x[order] for x in got)
        if t == STR:
            chars, size = _gather_text(pages, got[0], got[1])
            return {"": _room(chars, 200 * self.most), "_lens": _room(size.to(torch.int32), self.most),
                    "_valid": _room(got[2], self.most)}
        return {"": _room(got[0], self.most), "_valid": _room(got[1], self.most)}

    def __getitem__(self, name):
        if name == "rows":
            return int(self.result.num_rows)
        c, _, what = name[1:].partition("_")
        return self._column(int(c))["_" + what if what else ""]


class Batch(dict):
    """The rows of a batch's results: every plan's columns one after another, sorted as in Rows."""

    def __init__(self, results, state):
        self.results, self.state = results, state
        super().__init__(dict.fromkeys(["rows", "values", "valid"]))

    def __getitem__(self, name):
        if name == "rows":
            return torch.tensor([r.num_rows for r in self.results], dtype=torch.int64)
        out = []
        for r in self.results:
            fixed = [_fixed(t, p) for t, p in _columns(r)]
            order = _order(fixed)
            out += [f[0 if name == "values" else 1][order] for f in fixed]
        return _room(torch.cat(out), most_rows(self.state["case"]))


# ---- work ---------------------------------------------------------------------------------------------------------


def _bytes(t, n, null=0.0):
    if t == STR:
        return n * ((2 + 20) * (1 - null) + 0.125)
    return n * (WIDTH[t] * (1 - null) + 0.125)


def work(case):
    """Bytes of the columns' pages that the call reads, and of the pages that it writes."""
    kind = case["kind"]
    if kind == "filter":
        out = case["rows"] * case["keep"] * (1 - case["null"]) ** 2 * 0.84
        cols = [I32, I32, F64] + ([STR] if case["text"] else [])
        nulls = [0.0] + [case["null"]] * (len(cols) - 1)
        read = sum(_bytes(t, case["rows"], x) for t, x in zip(cols, nulls))
        return {"bytes": read + sum(_bytes(t, out) for t in cols), "flops": 0}
    if kind == "batch":
        total = 0.0
        for probe, builds in _chain_shapes(case):
            k = len(builds)
            total += (k + 1) * _bytes(I32, probe) + sum(2 * _bytes(I32, b) for b in builds)
            total += (2 * k + 1) * _bytes(I32, probe * (0.85 * 0.99) ** k)
        return {"bytes": total, "flops": 0}
    if kind == "star":
        kept = _star_kept(case)
        out = float(case["fact"])
        for keep in STAR_KEEP[:case["dims"]]:
            out *= keep
        read = (case["dims"] + 1) * _bytes(I32, case["fact"]) + 22 * out
        read += sum(_bytes(I32, k) + 22 * min(k, out) for k in kept)
        return {"bytes": read + out * (4 * (case["dims"] + 1) + 22 * (case["dims"] + 1)), "flops": 0}
    key, bt, ft = TYPES[case["key"]], TYPES[case["payload"]], TYPES[case["fact"]]
    out = case["probe"] * (1 - case["key_null"]) * (1 - case["outside"]) / (1 - case["dup"])
    read = _bytes(key, case["build"]) + _bytes(bt, case["build"], case["null"])
    read += _bytes(key, case["probe"], case["key_null"]) + _bytes(ft, case["probe"], case["null"])
    write = 2 * _bytes(key, out) + _bytes(bt, out, case["null"]) + _bytes(ft, out, case["null"])
    if STR in (bt, ft):
        read, write = read + _bytes(I32, case["probe"]), write + _bytes(I32, out)
    return {"bytes": read + write, "flops": 0}


def exact(case, seed):
    """None: a join and a filter pass values on and compute none; every output is a whole number or bytes."""
    return None
