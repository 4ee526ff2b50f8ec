"""Performance cases of the sort + group-by library.

Each case is one call (or one launch of a planned batch) through the public
binding, over inputs that are already on the GPU, at sizes taken from the
benchmark's configurations and the tests.  `listed()` names the cases,
`draw(rng)` gives further ones of the same ranges, `prepare(case, seed)` makes
the inputs, output buffers and plans a program keeps, `run(state)` is one
pass, `work(case)` the bytes a pass cannot do without, and `exact(case, seed)`
the floating results in plain torch.

Kinds
  sort_groupby  stable sort by one or two key columns, payload gather, and
                count / sum / min / max / mean per group (vdf_sort_groupby);
                full = False asks for the group table only
  materialize   argsort by one to three keys, then the gather of a frame's
                other columns through the permutation (vdf_sort_argsort,
                vdf_gather): the hard sort of a frame
  unique        keep mask of each key's first or last row (vdf_unique)
  join          left-join row matching (vdf_left_join_index)
  batch         many independent queries, planned once, one graph launch per
                pass (vdf_batch_*)
  csv           a delimited file's bytes into columns (vdf_csv_read)
"""
from __future__ import annotations

import math

import torch

import visondf_b200 as vdf
from visondf_b200 import datagen

DEV = "cuda:0"
_DT = {"i32": torch.int32, "i64": torch.int64, "u32": torch.uint32, "u64": torch.uint64, "f32": torch.float32,
       "f64": torch.float64}
_W = {"i32": 4, "i64": 8, "u32": 4, "u64": 8, "f32": 4, "f64": 8}
_SIGNED = {torch.uint32: torch.int32, torch.uint64: torch.int64}
_ORDER = {"asc": vdf.ORDER_ASC, "desc": vdf.ORDER_DESC_STABLE, "reverse": vdf.ORDER_DESC_REVERSE}

_context = None


def context() -> "vdf.Context":
    """The one context a program keeps."""
    global _context
    if _context is None:
        _context = vdf.Context(0)
    return _context


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest query of the batched and served configurations, sent
        # alone: one request for one small frame, where latency counts
        dict(name="query_1k", kind="sort_groupby", n=1_000, keys="i32", card=100, payload="f64,i64", nagg=2, full=True),
        # an ordinary small query with a wide key, of an odd size
        dict(name="query_60k_wide_key", kind="sort_groupby", n=60_001, keys="i64", card=9_000, payload="f64,i64",
             nagg=2, full=True),
        # the small configuration: a 1M-row frame, 10,000 int32 keys
        dict(name="frame_1m", kind="sort_groupby", n=1_000_000, keys="i32", card=10_000, payload="f64,i64", nagg=2,
             full=True),
        # two keys where the first ties (about two rows per value), odd size
        dict(name="two_keys_ties_9m", kind="sort_groupby", n=9_000_003, keys="i64,i32", card=4_500_000,
             payload="f64,i32,u64", nagg=2, full=True),
        # the headline configuration: 100M rows, full-range int64 key, Zipf int32 key
        dict(name="two_keys_100m", kind="sort_groupby", n=100_000_000, keys="i64,i32", card=0, payload="f64,i32,u64",
             nagg=2, full=True),
        # the group-by configuration at its two cardinalities; the group table
        # is what the caller wants
        dict(name="groupby_50m_keys_200m", kind="sort_groupby", n=200_000_000, keys="i64", card=50_000_000,
             payload="f64,i64", nagg=2, full=False),
        dict(name="groupby_16_keys_200m", kind="sort_groupby", n=200_000_000, keys="i32", card=16, payload="f64,i64",
             nagg=2, full=False),
        # the hard sort of a frame by a float column, descending: argsort and
        # materialize of five columns
        dict(name="sort_f64_frame_20m", kind="materialize", n=20_000_001, keys="f64", card=0, order="desc",
             cols="f64,i64,i32,f32,u64"),
        # de-duplication of an id column, and a fact table joined to a
        # dimension table a tenth its size (the benchmark's shapes)
        dict(name="unique_50m", kind="unique", n=50_000_000, keys="i64", card=25_000_000, last=False),
        dict(name="join_50m_5m", kind="join", n=50_000_000, right=5_000_000, keys="i64", method=0),
        # the batched configuration: 4,096 queries of 1k rows and up, one graph launch
        dict(name="batch_4096", kind="batch", queries=4096, megabytes=2048),
        # file ingest: the airline-shaped table
        dict(name="csv_256mb", kind="csv", megabytes=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["sort_groupby", "sort_groupby", "sort_groupby", "two_keys", "materialize", "unique", "join",
                       "batch", "csv"])
    if kind == "sort_groupby":
        n = _log(rng, 1_000, 150_000_000)
        return dict(kind=kind, n=n, keys=rng.choice(["i32", "i64"]), card=_log(rng, 2, max(2, n // 2)),
                    payload="f64,i64", nagg=2, full=n < 100_000_000 and rng.random() < 0.5)
    if kind == "two_keys":
        n = _log(rng, 1_000, 80_000_000)
        return dict(kind="sort_groupby", n=n, keys="i64,i32", card=rng.choice([0, max(1, n // 2)]),
                    payload="f64,i32,u64", nagg=2, full=True)
    if kind == "materialize":
        n = _log(rng, 1_000, 60_000_000)
        keys = [rng.choice(["i32", "i64", "u32", "u64", "f32", "f64"]) for _ in range(rng.choice([1, 1, 1, 2, 3]))]
        cols = [rng.choice(["i32", "i64", "f64", "u64", "f32"]) for _ in range(rng.randint(1, 5))]
        return dict(kind=kind, n=n, keys=",".join(keys), card=rng.choice([0, _log(rng, 2, max(2, n // 2))]),
                    order=rng.choice(["asc", "desc", "reverse"]), cols=",".join(cols))
    if kind == "unique":
        n = _log(rng, 1_000, 80_000_000)
        return dict(kind=kind, n=n, keys=rng.choice(["i32", "i64"]), card=_log(rng, max(2, n // 50), n),
                    last=rng.random() < 0.5)
    if kind == "join":
        n = _log(rng, 1_000, 80_000_000)
        return dict(kind=kind, n=n, right=max(1, n // rng.choice([2, 5, 10, 20])), keys=rng.choice(["i32", "i64"]),
                    method=rng.randint(0, 2))
    if kind == "batch":
        return dict(kind=kind, queries=_log(rng, 16, 4096), megabytes=_log(rng, 32, 1024))
    return dict(kind="csv", megabytes=_log(rng, 1, 400))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _full_range(n, dt, g):
    """n values over a dtype's whole range (N(0,1) for floats)."""
    if dt in ("f32", "f64"):
        return torch.randn(n, dtype=_DT[dt], device=DEV, generator=g)
    base = torch.int32 if _W[dt] == 4 else torch.int64
    t = torch.empty(n, dtype=base, device=DEV).random_(torch.iinfo(base).min, None, generator=g)
    return t if _DT[dt] == base else t.view(_DT[dt])


def _pick(pool, n, g):
    """n draws from a pool of values."""
    plain = pool.view(_SIGNED.get(pool.dtype, pool.dtype))
    t = plain[torch.randint(0, plain.numel(), (n,), device=DEV, generator=g)]
    return t.view(pool.dtype)


def _zipf(n, dt, g, ranks=1_000_000, s=1.1):
    """Zipf(s) over `ranks` random values, by inverse CDF."""
    w = torch.arange(1, ranks + 1, dtype=torch.float64, device=DEV) ** (-s)
    cdf = torch.cumsum(w, 0)
    cdf /= cdf[-1].clone()
    pool = _full_range(ranks, dt, g)
    out = torch.empty(n, dtype=pool.dtype, device=DEV)
    step = 1 << 24  # in pieces: the ranks are 8 bytes each
    for i in range(0, n, step):
        m = min(step, n - i)
        u = torch.rand(m, dtype=torch.float64, device=DEV, generator=g)
        out[i:i + m] = pool[torch.searchsorted(cdf, u, right=True).clamp_(max=ranks - 1)]
    return out


def _keys(case, g):
    n, card = case["n"], case["card"]
    out = []
    for k, dt in enumerate(case["keys"].split(",")):
        if case["kind"] == "sort_groupby" and k == 1:
            out.append(_zipf(n, dt, g))
        elif card == 0:
            out.append(_full_range(n, dt, g))
        elif card == 16 and case["kind"] == "sort_groupby":
            # two hot keys take 45 % of the rows each, the others share 10 %
            u = torch.rand(n, device=DEV, generator=g)
            i = torch.randint(2, card, (n,), device=DEV, generator=g)
            i[u < 0.9] = 0
            i[u < 0.45] = 1
            out.append(_full_range(card, dt, g)[i])
        else:
            out.append(_pick(_full_range(card, dt, g), n, g))
    return out


def _column(n, dt, k, g, wide):
    """A payload column: N(0,1) or lognormal floats, integers, row ids."""
    if dt in ("f64", "f32"):
        t = torch.randn(n, dtype=_DT[dt], device=DEV, generator=g)
        return t.exp_() if wide else t
    if dt == "i64":
        lo, hi = (0, 1 << 40) if wide else (-10**9, 10**9 + 1)
        return torch.randint(lo, hi, (n,), device=DEV, generator=g)
    if dt == "u64":
        return torch.arange(n, dtype=torch.int64, device=DEV).view(torch.uint64)
    return _full_range(n, dt, g)


def _payload(case, g):
    wide = not case["full"]  # the group-by configuration's value columns
    return [_column(case["n"], dt, k, g, wide) for k, dt in enumerate(case["payload"].split(","))]


def _frame(case, seed):
    g = _gen(seed)
    return _keys(case, g), _payload(case, g)


def _sides(case, seed):
    """Left and right join keys: three quarters of the left rows have a match."""
    g = _gen(seed)
    dt, nl, nr = case["keys"], case["n"], case["right"]
    right = _full_range(nr, dt, g)
    left = _pick(right, nl, g)
    miss = torch.rand(nl, device=DEV, generator=g) < 0.25
    left = torch.where(miss, _full_range(nl, dt, g), left)
    return left, right


def _specs(case):
    return datagen.batch_specs(nq=case["queries"], budget_bytes=case["megabytes"] << 20)


_AIRLINE_ROWS = 6_000  # rows of the block a file repeats


def _airline(case, seed):
    """(header, one block of rows, repeats) of an airline-shaped file."""
    data = datagen.airline_csv(target_bytes=1, seed_=int(seed) & 0x7FFFFFFF, block_rows=_AIRLINE_ROWS)
    cut = data.index(b"\n") + 1
    return data[:cut], data[cut:], max(1, (case["megabytes"] << 20) // (162 * _AIRLINE_ROWS))


def _clear(tensors, aggs):
    """Zeroes group buffers: slots past the last group stay as they are."""
    for t in tensors + [x for a in aggs for x in (a.sum, a.sum_hi, a.min, a.max, a.mean) if x is not None]:
        _plain(t).zero_()


def prepare(case, seed):
    kind = case["kind"]
    ctx = context()
    if kind == "sort_groupby":
        keys, pay = _frame(case, seed)
        aggs = list(range(case["nagg"]))
        full = case["full"]
        out = ctx.alloc_sort_groupby_outputs(keys, pay, aggs, True, full, full, full)
        _clear(out["gkeys"] + [out["count"]], out["aggs"])
        args = ctx.pack_sort_groupby(keys, pay, aggs, vdf.ORDER_ASC, True, out)
        return dict(kind=kind, keys=keys, pay=pay, out=out, args=args)
    if kind == "materialize":
        g = _gen(seed)
        n = case["n"]
        keys = _keys(case, g)
        cols = [_column(n, dt, k, g, False) for k, dt in enumerate(case["cols"].split(","))]
        return dict(kind=kind, keys=keys, cols=cols, order=_ORDER[case["order"]],
                    perm=torch.empty(n, dtype=torch.int32, device=DEV),
                    skeys=[torch.empty_like(k) for k in keys], out=[torch.empty_like(c) for c in cols])
    if kind == "unique":
        return dict(kind=kind, key=_keys(case, _gen(seed))[0], last=case["last"])
    if kind == "join":
        left, right = _sides(case, seed)
        return dict(kind=kind, left=left, right=right, method=case["method"])
    if kind == "batch":
        g = _gen(seed)
        queries = []
        for s in _specs(case):
            dt = "i64" if s["dtype"].__name__ == "int64" else "i32"
            key = _pick(_full_range(s["card"], dt, g), s["n"], g)
            queries.append((key, [_column(s["n"], "f64", 0, g, False), _column(s["n"], "i64", 1, g, False)]))
        out = vdf.Batch.alloc_outputs(sum(s["n"] for s in _specs(case)), [torch.float64, torch.int64], DEV)
        _clear([out["perm"], out["gkeys"], out["count"]], out["aggs"])
        return dict(kind=kind, batch=vdf.Batch(ctx, queries, outputs=out))
    header, block, reps = _airline(case, seed)
    rows = _AIRLINE_ROWS * reps
    # the caller's buffers for the four string columns (bytes, offsets)
    text = [(torch.zeros(40 * rows, dtype=torch.uint8, device=DEV),
             torch.zeros(rows + 1, dtype=torch.int64, device=DEV)) for _ in range(4)]
    h = torch.frombuffer(bytearray(header), dtype=torch.uint8).to(DEV)
    b = torch.frombuffer(bytearray(block), dtype=torch.uint8).to(DEV)
    return dict(kind="csv", data=torch.cat([h, b.repeat(reps)]), text=text)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _plain(t):
    """Unsigned columns as the signed type of their width (the same bytes)."""
    return t.view(_SIGNED.get(t.dtype, t.dtype))


def run(state):
    kind = state["kind"]
    ctx = context()
    if kind == "sort_groupby":
        ctx.sort_groupby_packed(state["args"])
        o = state["out"]
        res = {"groups": int(o["_ng"].value), "gkeys": [_plain(k) for k in o["gkeys"]], "count": o["count"],
               "aggs": [{"sum": a.sum, "sum_hi": a.sum_hi, "min": a.min, "max": a.max, "mean": a.mean}
                        for a in o["aggs"]]}
        if o["perm"] is not None:
            res.update(perm=o["perm"], keys=[_plain(k) for k in o["skeys"]], payload=[_plain(p) for p in o["pay"]])
        return res
    if kind == "materialize":
        ctx.argsort(state["keys"], state["order"], perm_out=state["perm"], sorted_keys_out=state["skeys"])
        ctx.gather(state["perm"], state["cols"], out=state["out"])
        return {"perm": state["perm"], "keys": [_plain(k) for k in state["skeys"]],
                "cols": [_plain(c) for c in state["out"]]}
    if kind == "unique":
        keep, count = ctx.unique(state["key"], keep_last=state["last"])
        return {"keep": keep, "count": count}
    if kind == "join":
        match, count = ctx.left_join_index(state["left"], state["right"], method=state["method"])
        return {"match": match, "count": count}
    if kind == "batch":
        b = state["batch"]
        b.launch_graph()
        return {"perm": b.perm, "gkeys": b.gkeys, "count": b.count, "n_groups": b.n_groups,
                "row_offset": b.row_offset, "group_offset": b.group_offset,
                "aggs": [{"sum": a.sum, "sum_hi": a.sum_hi, "min": a.min, "max": a.max, "mean": a.mean}
                         for a in b.aggs]}
    table = ctx.read_csv(state["data"], quote='"')
    cols, buffers = [], iter(state["text"])
    for k in range(table.ncol):
        if table.types[k] in ("s", "c"):
            text, offs = next(buffers)
            table.copy_column(k, text.data_ptr(), offs.data_ptr())
            cols += [text, offs]
        else:
            cols.append(_plain(table.view(k)))
    rows = table.nrow
    table.close()  # the views keep the memory until they are gone
    return {"rows": rows, "cols": cols}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _distinct(n, card):
    """Expected distinct values among n draws from card."""
    return n if card == 0 else card * -math.expm1(-n / card)


def _group_bytes(dts):
    """Bytes per group: count, and sum (sum_hi) / min / max / mean per column."""
    return 8 + sum((16 if dt[0] == "f" else 24) + 2 * _W[dt] for dt in dts)


def work(case):
    kind = case["kind"]
    if kind == "sort_groupby":
        n, keys, pay = case["n"], case["keys"].split(","), case["payload"].split(",")
        kw, pw = sum(_W[k] for k in keys), sum(_W[p] for p in pay)
        groups = n if len(keys) > 1 else _distinct(n, case["card"])
        rows = n * (kw + pw) + (n * (4 + kw + pw) if case["full"] else 0)
        return {"bytes": rows + groups * (kw + _group_bytes(pay[:case["nagg"]])), "flops": 0}
    if kind == "materialize":
        kw = sum(_W[k] for k in case["keys"].split(","))
        cw = sum(_W[c] for c in case["cols"].split(","))
        return {"bytes": case["n"] * (2 * kw + 4 + 2 * cw), "flops": 0}
    if kind == "unique":
        return {"bytes": case["n"] * (_W[case["keys"]] + 1), "flops": 0}
    if kind == "join":
        w = _W[case["keys"]]
        return {"bytes": case["n"] * (w + 4) + case["right"] * w, "flops": 0}
    if kind == "batch":
        total = 0.0
        for s in _specs(case):
            w = 8 if s["dtype"].__name__ == "int64" else 4
            total += s["n"] * (w + 16 + 4) + _distinct(s["n"], s["card"]) * (w + _group_bytes(["f64", "i64"]))
        return {"bytes": total, "flops": 0}
    # the file once, and per 162-byte row 15 doubles, 2 integers and 4 strings with their offsets
    size = case["megabytes"] << 20
    return {"bytes": size + size / 162 * (15 * 8 + 2 * 4 + 4 * 8 + 45), "flops": 0}


# ---------------------------------------------------------------------------
# the floating results in 64 bits
# ---------------------------------------------------------------------------
def _image(t, desc):
    """Signed integers in the order of a key column (floats by IEEE order)."""
    if t.dtype in (torch.float32, torch.float64):
        i = t.view(torch.int32 if t.dtype == torch.float32 else torch.int64)
        i = torch.where(i < 0, i ^ torch.iinfo(i.dtype).max, i)
    elif t.dtype in _SIGNED:
        i = t.view(_SIGNED[t.dtype])
        i = i ^ torch.iinfo(i.dtype).min
    else:
        i = t
    return ~i if desc else i


def _argsort(keys, order):
    perm = None
    for t in reversed(keys):
        i = _image(t, order == "desc")
        if perm is None:
            perm = torch.sort(i, stable=True)[1]
        else:
            perm = perm[torch.sort(i[perm], stable=True)[1]]
    return perm.flip(0) if order == "reverse" else perm


def _group_sums(v, gid, starts, g, n):
    """Sums per group of a sorted column, in f64."""
    if g <= 64:
        b = starts.tolist() + [n]
        return torch.stack([v[b[i]:b[i + 1]].double().sum() for i in range(g)])
    return torch.zeros(g, dtype=torch.float64, device=DEV).index_add_(0, gid, v.double())


def exact(case, seed):
    kind = case["kind"]
    if kind == "sort_groupby":
        keys, pay = _frame(case, seed)
        n = case["n"]
        perm = _argsort(keys, "asc")
        head = torch.zeros(n, dtype=torch.bool, device=DEV)
        head[0] = True
        for k in keys:
            s = k[perm]
            head[1:] |= s[1:] != s[:-1]
            del s
        starts = torch.nonzero(head).flatten()
        gid = torch.cumsum(head, 0).sub_(1)
        g = starts.numel()
        count = torch.diff(starts, append=torch.tensor([n], device=DEV)).double()
        aggs = []
        for p in pay[:case["nagg"]]:
            v = _plain(p)[perm]
            s = _group_sums(v, gid, starts, g, n)
            a = {"sum": None, "sum_hi": None, "min": None, "max": None, "mean": s / count}
            if v.dtype.is_floating_point:
                a["sum"] = s
                a["min"] = torch.full((g,), math.inf, dtype=v.dtype, device=DEV).scatter_reduce_(0, gid, v, "amin")
                a["max"] = torch.full((g,), -math.inf, dtype=v.dtype, device=DEV).scatter_reduce_(0, gid, v, "amax")
            aggs.append({k: None if x is None else torch.cat([x, x.new_zeros(n - g)]) for k, x in a.items()})
        res = {"groups": None, "gkeys": None, "count": None, "aggs": aggs}
        if case["full"]:
            res.update(perm=None, keys=None, payload=[p[perm] if p.dtype.is_floating_point else None for p in pay])
        return res
    if kind == "materialize":
        g = _gen(seed)
        keys = _keys(case, g)
        cols = [_column(case["n"], dt, k, g, False) for k, dt in enumerate(case["cols"].split(","))]
        if not any(t.dtype.is_floating_point for t in keys + cols):
            return None
        perm = _argsort(keys, case["order"])
        f = lambda ts: [t[perm] if t.dtype.is_floating_point else None for t in ts]  # noqa: E731
        return {"perm": None, "keys": f(keys), "cols": f(cols)}
    if kind == "csv":
        header, block, reps = _airline(case, seed)
        rows = [_fields(r) for r in block.decode().splitlines()]
        cols = []
        for k in range(len(rows[0])):
            if k < 2:
                cols.append(None)
            elif k < 6:
                cols += [None, None]
            else:
                cols.append(torch.tensor([float(r[k]) for r in rows], dtype=torch.float64, device=DEV).repeat(reps))
        return {"rows": None, "cols": cols}
    return None  # whole values only, or (batch) an arena whose layout is the plan's own


def _fields(line):
    """The fields of one record ('"' quotes a field with commas)."""
    out, cur, inside = [], [], False
    for ch in line:
        if ch == '"':
            inside = not inside
        elif ch == "," and not inside:
            out.append("".join(cur))
            cur = []
        else:
            cur.append(ch)
    out.append("".join(cur))
    return out
