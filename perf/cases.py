"""What a user of this framework has it do, as cases that can be measured.

Each case is one call (or one burst of requests) through the C ABI of include/ral/ral_c.h, with the
column descriptors a C++ caller keeps in hand.  Programs and queries belong to the case; the values
in the columns come from the seed.

  filter_project  a small or middling query: the fused LogicalFilter + LogicalProject of the plain
                  VM configuration, or of the twelve-operator projection behind a filter
  project         LogicalProject alone: the twelve-operator register program over five columns
  filter_gather   LogicalFilter alone: a predicate on one column, every column compacted
  gather          every column of a table by one index column (order-by, join, filter)
  aggregate       aggregations without GROUP BY over expressions
  text            a table scan over delimited text and its filter
  parquet         a table scan over a Parquet file in host memory and its filter
  batch           many programs over tables of uneven sizes in one launch
  served          a burst of filter + project requests over resident tables
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (_ROOT, os.path.join(_ROOT, "blazingdb-ral_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import ralgpu as R                     # noqa: E402
from ralgpu import dtypes as D         # noqa: E402
from ralgpu import workloads as W      # noqa: E402
from ralgpu.column import GdfColumn    # noqa: E402

DEV = "cuda"

AGGREGATE = ("LogicalAggregate(group=[{}], f1=[SUM(+(*($2, $3), /($2, $3)))], mn=[MIN(-($3, $2))], "
             "hits=[SUM(>($1, 0))], avg=[AVG($2)], mx=[MAX($4)], n=[COUNT($0)])")
# the lineitem-like scan: quantity, extendedprice, discount and shipdate, kept by TPC-H Q6's conditions
# or by quantity alone (about half of the rows)
TEXT_HALF = "LogicalFilter(condition=[<($0, 26)])"


def listed():
    return [
        # an interactive query over a dimension-sized table: the smallest call, all latency
        {"name": "filter_project_10k", "kind": "filter_project", "program": "plain_vm", "rows": 10_000, "selectivity": 0.0},
        # the plain VM configuration at its own size
        {"name": "filter_project_1m", "kind": "filter_project", "program": "plain_vm", "rows": 1_000_000, "selectivity": 0.0},
        # the headline projection at its own size
        {"name": "project_200m", "kind": "project", "rows": 200_000_000},
        # the same projection behind a filter that keeps half of the rows
        {"name": "filter_project_200m", "kind": "filter_project", "program": "fused", "rows": 200_000_000, "selectivity": 0.5},
        # a filter over a fact table: the largest scan / compaction / gather
        {"name": "filter_gather_500m", "kind": "filter_gather", "rows": 500_000_000, "selectivity": 0.5, "nulls": False},
        # an order-by of a whole table with nulls; a ragged row count
        {"name": "gather_permutation_100m", "kind": "gather", "rows": 99_999_989, "pattern": "permutation"},
        # a report's totals over a fact table; a ragged row count
        {"name": "aggregate_100m", "kind": "aggregate", "rows": 100_000_007},
        # TPC-H Q6's scan of 20M lines of text
        {"name": "text_20m", "kind": "text", "rows": 20_000_000, "query": "q6", "blank": 0.0},
        # the same scan over a Parquet file of PLAIN pages in page-locked memory
        {"name": "parquet_plain_6m", "kind": "parquet", "rows": 6_000_000, "dictionary": False, "optional": False,
         "locked": True, "query": "q6"},
        # dictionary-encoded pages with nulls, in ordinary host memory: half of the rows kept
        {"name": "parquet_dict_nulls_700k", "kind": "parquet", "rows": 700_001, "dictionary": True, "optional": True,
         "locked": False, "query": "half"},
        # the batched configuration, its tables capped at 1M rows
        {"name": "batch_256", "kind": "batch", "programs": 256, "cap": 1_000_000},
        # a burst of requests at the served configuration's table mix, up to 4M rows a table
        {"name": "served_16", "kind": "served", "requests": 16, "max_rows": 4_000_000},
    ]


def _log(rng, lo, hi):
    n = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    return n | 1 if rng.random() < 0.5 else n


def draw(rng):
    kind = rng.choice(["filter_project", "project", "filter_gather", "gather", "aggregate", "text", "parquet", "batch",
                       "served"])
    if kind == "filter_project":
        if rng.random() < 0.5:
            return {"kind": kind, "program": "plain_vm", "rows": _log(rng, 1e4, 1e7), "selectivity": 0.0}
        return {"kind": kind, "program": "fused", "rows": _log(rng, 1e4, 2e8),
                "selectivity": rng.choice([0.01, 0.1, 0.5, 0.9, 0.99])}
    if kind == "project":
        return {"kind": kind, "rows": _log(rng, 1e4, 2e8)}
    if kind == "filter_gather":
        return {"kind": kind, "rows": _log(rng, 1e4, 5e8), "selectivity": rng.choice([0.01, 0.5, 0.99]),
                "nulls": rng.random() < 0.5}
    if kind == "gather":
        return {"kind": kind, "rows": _log(rng, 1e4, 1e8), "pattern": rng.choice(["permutation", "random", "sorted"])}
    if kind == "aggregate":
        return {"kind": kind, "rows": _log(rng, 1e4, 2e8)}
    if kind == "text":
        return {"kind": kind, "rows": _log(rng, 1e4, 2e7), "query": rng.choice(["q6", "half", "all"]),
                "blank": rng.choice([0.0, 0.02])}
    if kind == "parquet":
        optional = rng.random() < 0.5
        return {"kind": kind, "rows": _log(rng, 1e4, 7e5 if optional else 6e6), "dictionary": rng.random() < 0.5,
                "optional": optional, "locked": rng.random() < 0.5, "query": rng.choice(["q6", "half", "all"])}
    if kind == "batch":
        return {"kind": kind, "programs": rng.randint(16, 256), "cap": _log(rng, 1e4, 1e6)}
    return {"kind": kind, "requests": rng.randint(4, 16), "max_rows": _log(rng, 1e5, 4e6)}


# ---- descriptors ------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _array(cols):
    structs = [c.to_c() for c in cols]
    arr = (C.POINTER(GdfColumn) * max(1, len(structs)))()
    for i, s in enumerate(structs):
        arr[i] = C.pointer(s)
    return arr, structs


def _zeros(dtype, n, with_valid=True):
    """An output column whose bytes are defined from the start."""
    data = torch.zeros(max(n, 1), dtype=D.torch_dtype(dtype), device=DEV)
    valid = torch.zeros(R.valid_alloc_size(max(n, 1)), dtype=torch.uint8, device=DEV) if with_valid else None
    return R.Column(data, valid, dtype, size=n)


def _check(rc):
    if rc:
        raise RuntimeError(R.lib().ral_last_error().decode())


def _outputs(outs, structs):
    """Every output's data and mask buffers, its row count and its null count (the rows past the
    count keep the zeros that the buffers were made with)."""
    r = []
    for c, s in zip(outs, structs):
        r.append(c.data)
        if c.valid is not None:
            r += [c.valid, int(s.null_count)]
        r.append(int(s.size))
    return r


def _padded(x, n):
    """x, then zeros up to n rows."""
    out = torch.zeros(n, dtype=x.dtype, device=x.device)
    out[:x.shape[0]] = x
    return out


def _columns(raw, n):
    return [R.Column(v, m, t, size=n, null_count=nn) for t, v, m, nn in raw]


def _unpacked(mask, n):
    """The first n bits of a packed mask as booleans (None: all set)."""
    if mask is None:
        return torch.ones(n, dtype=torch.bool, device=DEV)
    bits = (mask[:, None] >> torch.arange(8, dtype=torch.uint8, device=DEV)) & 1
    return bits.reshape(-1)[:n].bool()


# ---- filter (+ project), project, gather, aggregate --------------------------------------------

def _plain_vm(n, seed):
    """plain_vm's columns, generated on the GPU."""
    g = _generator(seed)
    c0 = torch.randint(0, 1_000_000, (n,), generator=g, device=DEV, dtype=torch.int64)
    c1 = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    c2 = torch.randint(1, 51, (n,), generator=g, device=DEV, dtype=torch.int32)
    c3 = torch.randint(0, 2400, (n,), generator=g, device=DEV, dtype=torch.int32)
    m, nulls = W.random_valid_mask(n, 0.10, g, DEV)
    return [(D.GDF_INT64, c0, None, 0), (D.GDF_FLOAT64, c1, m, nulls), (D.GDF_INT32, c2, None, 0),
            (D.GDF_DATE32, c3, None, 0)]


def _filter_project_raw(case, seed):
    n = case["rows"]
    return _plain_vm(n, seed) if case["program"] == "plain_vm" else W.fused_project_device(n, seed)


def _prepare_filter_project(case, seed):
    n = case["rows"]
    frame = _columns(_filter_project_raw(case, seed), n)
    if case["program"] == "plain_vm":
        fq, pq = W.PLAIN_VM_FILTER, W.PLAIN_VM_PROJECT
    else:
        fq, pq = W.filter_project_filter(case["selectivity"]), W.FILTER_PROJECT_PROJECT
    types, _ = R.project_output_types([c.dtype for c in frame], pq)
    outs = [_zeros(t, n) for t in types]
    fa, fs = _array(frame)
    oa, os_ = _array(outs)
    return dict(frame=frame, outs=outs, fa=fa, fs=fs, oa=oa, os=os_, fq=fq.encode(), pq=pq.encode(), n=C.c_int32(0))


def _run_filter_project(s):
    _check(R.lib().ral_filter_project(s["fa"], len(s["frame"]), s["fq"], s["pq"], s["oa"], len(s["outs"]), C.byref(s["n"])))
    return _outputs(s["outs"], s["os"])


def _fused_exact(raw):
    """f1, f2 and i1 of the twelve-operator projection for every row."""
    a, b, x, y, k = (v for _, v, _, _ in raw)
    f1 = x * y + x / y
    t5 = (y - x).abs()
    c = (b > 0).double()
    f2 = t5 + c * (x.floor() - t5)
    i1 = torch.fmod(a, k.long() + 1)
    return f1, f2, i1


def _exact_filter_project(case, seed):
    raw = _filter_project_raw(case, seed)
    n = case["rows"]
    if case["program"] == "plain_vm":
        (_, c0, _, _), (_, c1, m1, _), (_, c2, _, _), (_, c3, _, _) = raw
        v1 = _unpacked(m1, n)
        # a null operand makes the predicate null, and a null predicate drops the row
        keep = (((c2 >= 24) & (c1 < 0.05)) | (c0 % 7 == 3)) & (c3 < 1200) & v1
        f = (c1 * (1 - c1) + c2.double())[keep]
        return [_padded(f, n), None, None, None]
    keep = (raw[4][1] < round(1000 * case["selectivity"])) & _unpacked(raw[4][2], n)
    f1, f2, _ = _fused_exact(raw)
    return [_padded(f1[keep], n), None, None, None, _padded(f2[keep], n), None, None, None, None, None, None, None]


def _prepare_project(case, seed):
    n = case["rows"]
    spec = W.fused_project_program()
    cols = _columns(W.fused_project_device(n, seed), n)
    outs = [_zeros(t, n) for t in spec.output_dtypes]
    ia, is_ = _array(cols)
    oa, os_ = _array(outs)
    i16 = lambda v: np.ascontiguousarray(v, dtype=np.int16)    # noqa: E731
    i32 = lambda v: np.ascontiguousarray(v, dtype=np.int32)    # noqa: E731
    arrays = [i16(spec.left), i16(spec.right), i16(spec.outputs), i16(spec.final), i32(spec.ops), i32(spec.uops),
              i16(range(len(cols)))]
    p16, p32 = C.POINTER(C.c_int16), C.POINTER(C.c_int32)
    left, right, outp, final, ops, uops, idx = [a.ctypes.data_as(p16 if a.dtype == np.int16 else p32) for a in arrays]
    ls, rs = ((R.column.GdfScalar * len(spec.left))(*[R.Scalar(*x).to_c() for x in v]) for v in (spec.lscalars, spec.rscalars))
    args = (oa, len(outs), ia, len(cols), left, right, outp, len(spec.left), final, ops, uops, ls, rs, idx, len(cols))
    return dict(cols=cols, outs=outs, keep=(arrays, is_, os_), args=args)


def _run_project(s):
    _check(R.lib().ral_perform_operation(*s["args"]))
    return [t for c in s["outs"] for t in (c.data, c.valid)]


def _exact_project(case, seed):
    f1, f2, _ = _fused_exact(W.fused_project_device(case["rows"], seed))
    return [f1, None, f2, None, None, None]


def _prepare_filter_gather(case, seed):
    n = case["rows"]
    frame = _columns(W.filter_gather_device(n, seed, null_rate=0.05 if case["nulls"] else None), n)
    outs = [_zeros(c.dtype, n, c.valid is not None) for c in frame]
    fa, fs = _array(frame)
    oa, os_ = _array(outs)
    return dict(frame=frame, outs=outs, fa=fa, fs=fs, oa=oa, os=os_, n=C.c_int32(0),
                fq=W.filter_gather_query(case["selectivity"]).encode())


def _run_filter_gather(s):
    _check(R.lib().ral_process_filter(s["fa"], len(s["frame"]), s["fq"], s["oa"], C.byref(s["n"])))
    return _outputs(s["outs"], s["os"])


def _prepare_gather(case, seed):
    n = case["rows"]
    frame = _columns(W.filter_gather_device(n, seed, null_rate=0.05), n)
    g = _generator(seed + 1)
    if case["pattern"] == "permutation":
        idx = torch.randperm(n, generator=g, device=DEV, dtype=torch.int32)
    else:
        idx = torch.randint(0, n, (n,), generator=g, device=DEV, dtype=torch.int32)
        if case["pattern"] == "sorted":
            idx = torch.sort(idx).values
    icol = R.Column(idx, None, D.GDF_INT32, n)
    outs = [_zeros(c.dtype, n) for c in frame]
    fa, fs = _array(frame)
    oa, os_ = _array(outs)
    return dict(frame=frame, outs=outs, fa=fa, fs=fs, oa=oa, os=os_, icol=icol, ic=icol.to_c())


def _run_gather(s):
    _check(R.lib().ral_materialize_columns(C.cast(s["fa"], C.c_void_p), C.cast(s["oa"], C.c_void_p), len(s["frame"]),
                                           C.byref(s["ic"])))
    return _outputs(s["outs"], s["os"])


def _prepare_aggregate(case, seed):
    n = case["rows"]
    frame = _columns(W.fused_project_device(n, seed), n)
    fa, fs = _array(frame)
    return dict(frame=frame, fa=fa, fs=fs, res=(R.column.GdfScalar * 16)(), n=C.c_int32(0), q=AGGREGATE.encode())


def _run_aggregate(s):
    _check(R.lib().ral_process_aggregate(C.cast(s["fa"], C.c_void_p), len(s["frame"]), s["q"], s["res"], 16, C.byref(s["n"])))
    return [R.Scalar.from_c(s["res"][i]).value for i in range(s["n"].value)]


def _exact_aggregate(case, seed):
    raw = W.fused_project_device(case["rows"], seed)
    n = case["rows"]
    x, y = raw[2][1], raw[3][1]
    valid = _unpacked(raw[2][2], n)
    # an evaluated input counts every row, a bare column its valid rows
    return [float((x * y + x / y).sum()), float((y - x).min()), None, float(x[valid].sum() / valid.sum()), None, None]


# ---- table scans ------------------------------------------------------------------------------

def _query(case):
    return {"q6": W.TEXT_FILTER, "half": TEXT_HALF, "all": None}[case["query"]]


def _lineitem(n, g):
    """The lineitem-like draws of the workloads module, on the GPU: orderkey, partkey, quantity,
    extendedprice in cents, discount and tax in hundredths, shipdate and commitdate in days."""
    def ints(lo, hi):
        return torch.randint(lo, hi, (n,), generator=g, device=DEV, dtype=torch.int64)
    ship = ints(8036, 10591)
    return [ints(1, 6_000_000_000), ints(1, 2_000_000), ints(1, 51), ints(90000, 10500000), ints(0, 11), ints(0, 9),
            ship, ship + ints(-60, 60)]


def _civil(days):
    """Year, month and day of days since 1970-01-01."""
    z = days + 719468
    era = z // 146097
    doe = z - era * 146097
    yoe = (doe - doe // 1460 + doe // 36524 - doe // 146096) // 365
    doy = doe - (365 * yoe + yoe // 4 - yoe // 100)
    mp = (5 * doy + 2) // 153
    d = doy - (153 * mp + 2) // 5 + 1
    m = mp + torch.where(mp < 10, 3, -9)
    return yoe + era * 400 + (m <= 2).long(), m, d


def _text(n, seed, blank):
    """n lines of '|'-delimited lineitem-like text (numbers without leading zeros), and for each of
    the eight fields its blank rows (None: none)."""
    g = _generator(seed)
    v = _lineitem(n, g)
    cells, shown = [], []            # one column of bytes each, and whether a line has it

    def put(b, on=None):
        cells.append(b)
        shown.append(on)

    def number(x, width, padded, on):
        for k in range(width - 1, -1, -1):
            p = 10 ** k
            lead = on if padded or k == 0 else (x >= p if on is None else on & (x >= p))
            put((x // p % 10 + 48).to(torch.uint8), lead)

    def const(ch, on=None):
        put(torch.full((n,), ord(ch), dtype=torch.uint8, device=DEV), on)

    blanks = []
    for f in range(8):
        on = None
        if blank > 0:
            on = torch.rand(n, generator=g, device=DEV) >= blank
            blanks.append(~on)
        else:
            blanks.append(None)
        if f < 3:
            number(v[f], (10, 7, 2)[f], False, on)
        elif f == 3:
            number(v[f] // 100, 6, False, on)
            const(".", on)
            number(v[f] % 100, 2, True, on)
        elif f < 6:
            number(v[f] // 100, 1, False, on)
            const(".", on)
            number(v[f] % 100, 2, True, on)
        else:
            y, m, d = _civil(v[f])
            number(y, 4, True, on)
            const("-", on)
            number(m, 2, True, on)
            const("-", on)
            number(d, 2, True, on)
        const("|" if f < 7 else "\n")
    wide = torch.stack(cells, dim=1)
    del cells
    mask = torch.ones_like(wide, dtype=torch.bool)
    for j, on in enumerate(shown):
        if on is not None:
            mask[:, j] = on
    return wide[mask], v, blanks


def _scan_values(v):
    """The projected columns' values (quantity, extendedprice, discount, shipdate in milliseconds)."""
    return [v[2].int(), v[3].double() / 100.0, v[4].double() / 100.0, v[6] * 86_400_000]


def _scan_keep(case, v, blanks):
    """The rows that the case's filter keeps: its conditions hold and none of their columns is null."""
    keep = torch.ones_like(v[2], dtype=torch.bool)
    used = ()
    if case["query"] == "q6":
        # 1994-01-01 <= shipdate < 1995-01-01 and 0.05 <= discount <= 0.07 and quantity < 24
        keep = (v[6] >= 8766) & (v[6] < 9131) & (v[4] >= 5) & (v[4] <= 7) & (v[2] < 24)
        used = (2, 4, 6)
    elif case["query"] == "half":
        keep = v[2] < 26
        used = (2,)
    for f in used:
        if blanks[f] is not None:
            keep = keep & ~blanks[f]
    return keep


def _exact_scan(case, v, blanks):
    keep = _scan_keep(case, v, blanks)
    out = []
    for x, f in zip(_scan_values(v), W.TEXT_PROJECTIONS):
        x = x.masked_fill(blanks[f], 0) if blanks[f] is not None else x
        out += [_padded(x[keep], case["rows"]) if x.dtype == torch.float64 else None, None, None, None]
    return out


def _scan_outputs(n):
    outs = [_zeros(W.TEXT_DTYPES[c], n) for c in W.TEXT_PROJECTIONS]
    oa, os_ = _array(outs)
    return outs, oa, os_, (C.c_int32 * 4)(*W.TEXT_PROJECTIONS)


def _prepare_text(case, seed):
    n = case["rows"]
    text, _, _ = _text(n, seed, case["blank"])
    outs, oa, os_, pr = _scan_outputs(n)
    q = _query(case)
    return dict(text=text, outs=outs, oa=oa, os=os_, pr=pr, rows=n, q=q.encode() if q else None, n=C.c_int32(0),
                fd=(C.c_int32 * len(W.TEXT_DTYPES))(*W.TEXT_DTYPES))


def _run_text(s):
    for o in s["os"]:
        o.size = s["rows"]           # the capacity; the call leaves the rows kept
    _check(R.lib().ral_text_scan_filter(s["text"].data_ptr(), s["text"].numel(), b"|", b"\n", 0, s["fd"], len(s["fd"]),
                                        s["pr"], 4, s["q"], C.cast(s["oa"], C.c_void_p), C.byref(s["n"])))
    return _outputs(s["outs"], s["os"])


def _exact_text(case, seed):
    _, v, blanks = _text(case["rows"], seed, case["blank"])
    return _exact_scan(case, v, blanks)


def _parquet_values(case, seed):
    g = _generator(seed)
    v = _lineitem(case["rows"], g)
    blanks = [None] * 8
    if case["optional"]:
        # quantity and discount are nullable, with 3% nulls
        for f in (2, 4):
            blanks[f] = torch.rand(case["rows"], generator=g, device=DEV) < 0.03
    return v, blanks


def _prepare_parquet(case, seed):
    n = case["rows"]
    v, blanks = _parquet_values(case, seed)
    cols = []
    for x, f in zip(_scan_values(v), W.TEXT_PROJECTIONS):
        valid = None if blanks[f] is None else (~blanks[f]).cpu().numpy()
        cols.append((W.LINEITEM_NAMES[f], W.TEXT_DTYPES[f], x.cpu().numpy(), valid))
    blob = W.parquet_bytes(cols, dictionary=case["dictionary"])
    host = torch.frombuffer(bytearray(blob), dtype=torch.uint8)
    if case["locked"]:
        host = host.pin_memory()
    outs, oa, os_, _ = _scan_outputs(n)
    q = _query(case)
    return dict(file=host, outs=outs, oa=oa, os=os_, pr=(C.c_int32 * 4)(0, 1, 2, 3), rows=n, q=q.encode() if q else None,
                n=C.c_int32(0))


def _run_parquet(s):
    for o in s["os"]:
        o.size = s["rows"]
    _check(R.lib().ral_parquet_scan_filter(C.c_void_p(s["file"].data_ptr()), s["file"].numel(), s["pr"], 4, s["q"],
                                           C.cast(s["oa"], C.c_void_p), C.byref(s["n"])))
    return _outputs(s["outs"], s["os"])


def _exact_parquet(case, seed):
    v, blanks = _parquet_values(case, seed)
    return _exact_scan(case, v, blanks)


# ---- many programs ----------------------------------------------------------------------------

def _batch_tables(case):
    mix = W.batched_mix(case["programs"])
    for t in mix:
        t.rows = min(t.rows, case["cap"])
    return mix


def _prepare_batch(case, seed):
    mix = _batch_tables(case)
    plans = [R.parse_project_plan(t.dtypes, t.project) for t in mix]
    # one buffer per output type, each column at a 64-byte boundary; one buffer for all masks
    place, used = [], {}
    for t, pp in zip(mix, plans):
        for dt in pp["evaluated_dtypes"]:
            td = D.torch_dtype(dt)
            at, mat = used.get(td, 0), used.get("mask", 0)
            place.append((td, at, mat))
            used[td] = at + (t.rows + 63) // 64 * 64
            used["mask"] = mat + R.valid_alloc_size(t.rows)
    data = {td: torch.zeros(k, dtype=td, device=DEV) for td, k in used.items() if td != "mask"}
    masks = torch.zeros(used["mask"], dtype=torch.uint8, device=DEV)
    batch = R.Batch()
    at = iter(place)
    for i, (t, pp) in enumerate(zip(mix, plans)):
        t.seed = (int(seed) * 1_000_003 + i) % (1 << 31)
        cols = _columns(W.batched_table_device(t, DEV), t.rows)
        outs = []
        for dt in pp["evaluated_dtypes"]:
            td, d0, m0 = next(at)
            outs.append(R.Column(data[td][d0:d0 + t.rows], masks[m0:m0 + R.valid_alloc_size(t.rows)], dt, size=t.rows))
        batch.add(outs, [cols[c] for c in pp["input_columns"]], pp["left"], pp["right"], pp["outputs"],
                  pp["final_output_positions"], pp["operators"], pp["unary_operators"], pp["left_scalars"],
                  pp["right_scalars"])
    batch.prepare()
    return dict(batch=batch, data=data, masks=masks)


def _run_batch(s):
    s["batch"].run()
    return {"data": {str(k): v for k, v in s["data"].items()}, "masks": s["masks"]}


def _served(case):
    """Eight tables and two queries a table, each query two expressions of the served mix."""
    tables = W.served_tables(8, max_rows=float(case["max_rows"]))
    rng = np.random.default_rng(W.SEED + 5)
    queries = []
    for q in range(16):
        dts = tables[q % 8].dtypes
        exprs = ", ".join(f"e{i}=[{W.random_rex(rng, int(rng.integers(1, 8)), len(dts))}]" for i in range(2))
        queries.append((q % 8, f"LogicalFilter(condition=[{W.random_predicate(rng, int(rng.integers(1, 6)), dts)}])",
                        f"LogicalProject({exprs})"))
    return tables, queries


def _prepare_served(case, seed):
    tables, queries = _served(case)
    srv = R.Server(budget_bytes=16 << 30)
    ids = []
    for i, t in enumerate(tables):
        t.seed = (int(seed) * 1_000_003 + i) % (1 << 31)
        ids.append(srv.add_table(_columns(W.served_table_device(t, DEV), t.rows)))
    qids = [srv.add_query(ids[t], f, p) for t, f, p in queries]
    outs = []
    for q, (t, _, _) in list(zip(qids, queries))[:case["requests"]]:
        outs.append([_zeros(dt, tables[t].rows) for dt in srv.query_outputs(q)[0]])
    torch.cuda.synchronize()
    srv.start()
    return dict(srv=srv, requests=[(q, o, *_array(o)) for q, o in zip(qids, outs)])


def _run_served(s):
    srv = s["srv"]
    rids = [srv.submit(q, keep=True) for q, _, _, _ in s["requests"]]
    out = []
    for rid, (_, cols, arr, _) in zip(rids, s["requests"]):
        srv.wait(rid)
        _check(R.lib().ral_server_copy_result(srv._h, rid, arr, len(cols)))
        srv.release(rid)
        out += [t for c in cols for t in (c.data, c.valid)]
    return out


# ---- the interface ----------------------------------------------------------------------------

def prepare(case, seed):
    return case["kind"], globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state[0]](state[1])


def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    return f(case, seed) if f else None


def _plain_vm_kept():
    """Share of rows that the plain VM filter keeps: its conditions are independent."""
    return 0.9 * 0.5 * (1 - (1 - 0.05 * 27 / 50) * (1 - 1 / 7))


def work(case):
    n = case.get("rows", 0)
    k = case["kind"]
    if k == "filter_project":
        if case["program"] == "plain_vm":
            return {"bytes": n * (8 + 8.125 + 4 + 4) + n * _plain_vm_kept() * 8.125, "flops": 12 * n}
        s = case["selectivity"] * 0.95
        # the filter's column whole; the others where rows are kept
        return {"bytes": n * 4.125 + s * n * 32.5 + s * n * 24.375, "flops": n + 12 * s * n}
    if k == "project":
        return {"bytes": n * (36.625 + 24.375), "flops": 12 * n}
    if k == "filter_gather":
        s = case["selectivity"] * (0.95 if case["nulls"] else 1.0)
        m = 0.125 if case["nulls"] else 0.0
        return {"bytes": n * (4 + m) + s * n * (25 + 5 * m) + s * n * (29 + 6 * m), "flops": n}
    if k == "gather":
        return {"bytes": n * (4 + 2 * 29 + 12 * 0.125), "flops": 0}
    if k == "aggregate":
        return {"bytes": n * (8 + 8.125 + 8 + 4.125), "flops": 8 * n}
    if k in ("text", "parquet"):
        kept = {"q6": 365 / 2555 * 3 / 11 * 23 / 50, "half": 0.5, "all": 1.0}[case["query"]]
        if k == "text":
            # the mean line: 9.8 + 6.9 + 1.8 + 7.8 + 4 + 4 + 10 + 10 characters and eight separators
            size = n * 62.4 * (1 - 0.85 * case["blank"])
        elif case["dictionary"]:
            # quantity 6 bits, extendedprice PLAIN, discount 4 bits, shipdate 12 bits
            size = n * (8 + 22 / 8) + (n / 4 if case["optional"] else 0)
        else:
            size = n * 28 + (n / 4 if case["optional"] else 0)
        return {"bytes": size + n * kept * 28.5, "flops": 0}
    if k == "batch":
        b = f = 0
        for t in _batch_tables(case):
            pp = R.parse_project_plan(t.dtypes, t.project)
            b += t.rows * sum(D.WIDTH[t.dtypes[c]] + (0.125 if t.null_rates[c] > 0 else 0) for c in pp["input_columns"])
            b += t.rows * sum(D.WIDTH[dt] + 0.125 for dt in pp["evaluated_dtypes"])
            f += t.rows * t.n_ops
        return {"bytes": b, "flops": f}
    tables, queries = _served(case)
    b = f = 0
    for t, fq, pq in queries[:case["requests"]]:
        used = {int(c) for c in "".join(ch if ch.isdigit() or ch == "$" else " " for ch in fq + pq).replace("$", " $").split()
                if c.startswith("$") for c in [c[1:]]}
        types, _ = R.project_output_types(tables[t].dtypes, pq)
        b += tables[t].rows * (sum(D.WIDTH[tables[t].dtypes[c]] + 0.125 for c in used) + 0.5 * sum(D.WIDTH[x] + 0.125 for x in types))
        f += tables[t].rows * 12
    return {"bytes": b, "flops": f}
