"""The work that is timed: what users of the engine have it do, through its public entry points.

Three kinds of call are covered, each over the range of sizes, key shapes and types it is used with:

  groupby    ``GroupBy(keys).aggregate(requests)`` on device columns: dense and sparse integer ids, composite keys,
             STRING and FLOAT64 keys, uniform and Zipf-distributed groups, masks on keys and values, both null policies
  partition  ``hash_partition(table, ...)``: the step in front of a shuffle between GPUs
  stream     ``StreamingGroupBy``: batches folded into a persistent state, then finalized

The five benchmark configurations (C1-C5 of ``workloads.py``) are among the cases at their full sizes.  Their data is
generated on the GPU here, with other seeds than there.

The order of the groups in a result (and of the rows inside a partition) is unspecified, so two correct runs differ in
it.  ``run`` returns the result columns as they are; the mapping that holds them (``InOrder``) puts the rows into a
defined order at the moment somebody reads them, which is not part of the work a user has done.
"""
import math

import numpy as np
import torch

import cudf_b200 as cb
from cudf_b200.aggregation import Aggregation
from cudf_b200.partition import hash_partition
from cudf_b200.types import Kind, NullPolicy, STORAGE_DTYPE, TypeId, result_type, type_width

KINDS = {"sum": Kind.SUM, "count": Kind.COUNT_VALID, "mean": Kind.MEAN, "min": Kind.MIN, "max": Kind.MAX,
         "var": Kind.VARIANCE, "std": Kind.STD}
DTYPES = {"i8": torch.int8, "i16": torch.int16, "i32": torch.int32, "i64": torch.int64, "f32": torch.float32,
          "f64": torch.float64}
TYPE_IDS = {"i8": TypeId.INT8, "i16": TypeId.INT16, "i32": TypeId.INT32, "i64": TypeId.INT64, "f32": TypeId.FLOAT32,
            "f64": TypeId.FLOAT64, "str": TypeId.STRING}
MEAN_STRING = 20   # lengths are uniform in 8..32


def _groupby(rows, keys, groups, values, aggs, skew="uniform", ids="dense", key_nulls=0.0, nulls=0.0, policy="exclude",
             dropna=False):
    return {"do": "groupby", "rows": rows, "keys": keys, "groups": groups, "values": values, "aggs": aggs, "skew": skew,
            "ids": ids, "key_nulls": key_nulls, "nulls": nulls, "policy": policy, "dropna": dropna}


def listed():
    return [
        # the smallest calls: a filtered or interactive frame of a thousand rows, where only latency counts
        {"name": "tiny", **_groupby(1000, "i32", 50, "f64", "sum,count,mean")},
        # C1: the usual small report, one integer key, sums and means of a nullable column
        {"name": "c1", **_groupby(10_000_000, "i64", 1000, "f64", "sum,count,mean", nulls=0.05)},
        # C2: dropna() and the mean over a composite key of 10K groups
        {"name": "c2", **_groupby(100_000_000, "i32,i32", 10_000, "f32", "mean", nulls=0.02, dropna=True)},
        # a summary by a category column: few groups, so that many rows meet on each, integer values
        {"name": "categories", **_groupby(50_000_000, "i32", 64, "i64", "sum,min,max,mean")},
        # per-user statistics: ids that are spread over 64 bits, more groups than a small table holds
        {"name": "users", **_groupby(20_000_003, "i64", 200_000, "f64", "mean,var", ids="sparse", nulls=0.01)},
        # C3: nearly as many groups as there can be, exact integer results
        {"name": "c3", **_groupby(500_000_000, "i64", 100_000_000, "i64", "sum,min,max,count")},
        # C4: a heavily skewed id column (events per user, words per corpus)
        {"name": "c4", **_groupby(1_000_000_000, "i64", 10_000_000, "f64", "sum,mean,var", skew="zipf", nulls=0.01)},
        # C5: strings and an integer as the key, every usual aggregation of two columns
        {"name": "c5", **_groupby(200_000_000, "str,i32", 16_000_000, "f64,i32", "sum,count,mean,min,max", nulls=0.03)},
        # a string key in a frame of ordinary size (names, urls), ragged row count
        {"name": "names", **_groupby(1_000_003, "str", 50_000, "i32", "count,min,max,sum", nulls=0.03)},
        # a composite key wider than 64 bits, nulls kept as a group, two value columns
        {"name": "wide", **_groupby(5_000_003, "i64,i32", 100_000, "f64,i32", "sum,mean,max", key_nulls=0.02, nulls=0.03,
                                    policy="include")},
        # the shuffle's pre-step: rows with a nullable and a narrow column into the partitions of 8 ranks
        {"name": "partition", "do": "partition", "rows": 100_000_000, "keys": "i64", "columns": "f64,i32", "groups": 10_000_000,
         "nulls": 0.05, "parts": 8},
        # a feed that arrives in batches
        {"name": "stream", "do": "stream", "batches": 16, "rows": 1_000_000, "keys": "i64", "groups": 100_000, "values": "f64",
         "aggs": "sum,count,mean,max", "nulls": 0.03},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choices(["packed", "string", "wide", "partition", "stream"], [10, 3, 2, 3, 2])[0]
    nulls = rng.choice([0.0, 0.0, 0.01, 0.05, 0.3])
    if what == "partition":
        return {"do": "partition", "rows": _log_uniform(rng, 1_000, 200_000_000), "keys": rng.choice(["i64", "i32", "i64,i32"]),
                "columns": rng.choice(["f64", "f64,i32", "f32", "i64,i16,f64", "i8"]), "groups": _log_uniform(rng, 10, 50_000_000),
                "nulls": nulls, "parts": rng.choice([2, 3, 4, 8, 8, 8, 16, 64, 200])}
    if what == "stream":
        return {"do": "stream", "batches": rng.randint(2, 16), "rows": _log_uniform(rng, 1_000, 4_000_000),
                "keys": rng.choice(["i64", "i32", "i32,i32", "str"]), "groups": _log_uniform(rng, 10, 1_000_000),
                "values": rng.choice(["f64", "i64", "f32", "f64,i32"]), "aggs": rng.choice(["sum,count,mean,max", "mean", "sum,count"]),
                "nulls": nulls}
    one = rng.choice(["f64", "f32", "i64", "i32"])
    aggs = rng.choice(["sum,count,mean", "mean", "sum,min,max,count", "sum,mean,var", "min,max,mean", "count", "std"])
    if what == "string":
        rows = _log_uniform(rng, 1_000, 100_000_000)
        return _groupby(rows, rng.choice(["str", "str", "str,i32"]), min(rows, _log_uniform(rng, 10, 8_000_000)),
                        rng.choice([one, "f64,i32"]), aggs, nulls=nulls)
    if what == "wide":
        rows = _log_uniform(rng, 1_000, 20_000_000)
        return _groupby(rows, rng.choice(["i64,i32", "i64,i64", "f64", "f64,i32"]), min(rows, _log_uniform(rng, 10, 2_000_000)),
                        rng.choice([one, "f64,i32"]), aggs, key_nulls=rng.choice([0.0, 0.02]), nulls=nulls,
                        policy=rng.choice(["exclude", "include"]))
    rows = _log_uniform(rng, 1_000, 300_000_000)
    two = rows <= 100_000_000 and rng.random() < 0.3
    return _groupby(rows, rng.choice(["i64", "i64", "i32", "i32,i32", "i16,i32"]), min(rows, _log_uniform(rng, 4, 50_000_000)),
                    "f64,i32" if two else one, aggs, skew=rng.choice(["uniform", "uniform", "uniform", "zipf"]),
                    ids=rng.choice(["dense", "dense", "sparse"]), key_nulls=rng.choice([0.0, 0.0, 0.0, 0.02]), nulls=nulls,
                    policy=rng.choice(["exclude", "exclude", "include"]), dropna=nulls > 0 and rng.random() < 0.25)


# ---------------------------------------------------------------------------------------------------- inputs
# Which group a row belongs to and which rows are null follow from a counter-based generator over the row numbers, turned
# by an amount that the seed decides: inputs of different seeds differ in every row, but hold the same number of groups,
# so that their results have the same shape.  Values, strings and the labels of skewed groups come from the seed.
CHUNK = 96_000_000   # rows whose temporaries are alive together (a multiple of 32)


class _Rows:
    """Random words for the rows of one table: ``bits(stream, lo, hi)`` for rows lo..hi."""

    def __init__(self, n, gen, table=0):
        self.n, self.gen, self.table = n, gen, table
        self.turn = int(torch.randint(0, n, (1,), device="cuda", generator=gen))

    def bits(self, stream, lo, hi):
        h = (torch.arange(lo, hi, dtype=torch.int64, device="cuda") + self.turn) % self.n
        h += (self.table * 64 + stream + 1) * 0x632BE59BD9B4E019 % (1 << 62)
        for shift, mult in ((32, -3335678366873096957), (29, -8378864009470890807)):   # (odd multipliers)
            h ^= (h >> shift) & ((1 << (64 - shift)) - 1)
            h *= mult
        return h ^ ((h >> 32) & 0xFFFFFFFF)

    def uniform(self, stream, lo, hi):
        return ((self.bits(stream, lo, hi) >> 11) & ((1 << 53) - 1)).to(torch.float64) * 2.0 ** -53


def _column(t, frac, rows, stream):
    """A column over `t` with `frac` of its rows null (bitmask words LSB first, 64 bytes of padding)."""
    if frac <= 0:
        return cb.Column.from_tensor(t)
    n = rows.n
    words = torch.zeros((n + 31) // 32 + 16, dtype=torch.int32, device="cuda")
    shifts = torch.arange(32, dtype=torch.int32, device="cuda")
    valid_rows = 0
    for lo in range(0, n, CHUNK):
        hi = min(n, lo + CHUNK)
        bits = torch.zeros((hi - lo + 31) // 32 * 32, dtype=torch.bool, device="cuda")
        bits[:hi - lo] = rows.uniform(stream, lo, hi) >= frac
        valid_rows = valid_rows + bits.sum()
        words[lo // 32: (hi + 31) // 32] = (bits.view(-1, 32).to(torch.int32) << shifts).sum(1, dtype=torch.int32)
    return cb.Column.from_tensor(t, words, null_count=n - int(valid_rows))


def _group_ids(rows, stream, groups, skew):
    out = torch.empty(rows.n, dtype=torch.int64, device="cuda")
    if skew == "zipf":   # in whole numbers, which add up to the same sums every time
        cdf = torch.cumsum((torch.arange(1, groups + 1, device="cuda", dtype=torch.float64) ** -1.1 * 2.0 ** 44).to(torch.int64), 0)
        total = int(cdf[-1])
        label = torch.randperm(groups, device="cuda", generator=rows.gen)
    for lo in range(0, rows.n, CHUNK):
        hi = min(rows.n, lo + CHUNK)
        if skew == "zipf":
            out[lo:hi] = label[torch.searchsorted(cdf, (rows.uniform(stream, lo, hi) * total).to(torch.int64), right=True)]
        else:
            out[lo:hi] = ((rows.bits(stream, lo, hi) >> 1) & 0x7FFFFFFFFFFFFFFF) % groups
    return out


def _strings(ids, pool, gen):
    """STRING column of a pool's strings at `ids`: [a-z0-9], lengths spread over 8..32; five characters tell a pool's strings apart."""
    n = ids.numel()
    at = torch.arange(pool, dtype=torch.int64, device="cuda")
    plen = 8 + (at * 7919 + 13) % 25
    poff = torch.zeros(pool + 1, dtype=torch.int64, device="cuda")
    poff[1:] = torch.cumsum(plen, 0)
    alphabet = torch.tensor(list(b"abcdefghijklmnopqrstuvwxyz0123456789"), dtype=torch.uint8, device="cuda")
    pchars = alphabet[torch.randint(0, 36, (int(poff[-1]),), device="cuda", generator=gen)]
    code = (at * 30233089 + 17) % 36 ** 5
    for d in range(5):
        pchars[poff[:-1] + 1 + d] = alphabet[code % 36]
        code = code // 36
    lens = plen[ids]
    offs = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    offs[1:] = torch.cumsum(lens, 0)
    total = int(offs[-1])
    chars = torch.empty(total, dtype=torch.uint8, device="cuda")
    for lo in range(0, n, CHUNK // 5):
        hi = min(n, lo + CHUNK // 5)
        b0, b1 = int(offs[lo]), int(offs[hi])
        src = torch.repeat_interleave(poff[ids[lo:hi]] - offs[lo:hi], lens[lo:hi]) + torch.arange(b0, b1, device="cuda")
        chars[b0:b1] = pchars[src]
    large = total > 0x7FFFFFFF
    o = offs if large else offs.to(torch.int32)
    return cb.Column(TypeId.STRING, n, chars, None, 0, 0, o.view(torch.uint8), TypeId.INT64 if large else TypeId.INT32)


def _key_domains(keys, groups):
    """Distinct values of every key column so that their combinations number about `groups`."""
    kinds = keys.split(",")
    if len(kinds) == 1:
        return [groups]
    if kinds[0] == "str":
        return [max(1, groups // 16), 16]
    first = max(1, int(round(math.sqrt(groups))))
    if kinds[0] == "i16":
        first = min(first, 10_000)
    return [first, max(1, groups // first)]


def _key_columns(case, rows, seed):
    cols = []
    for i, (kind, dom) in enumerate(zip(case["keys"].split(","), _key_domains(case["keys"], case["groups"]))):
        ids = _group_ids(rows, 2 * i, dom, case.get("skew", "uniform"))
        if kind == "str":
            cols.append(_strings(ids, dom, torch.Generator(device="cuda").manual_seed(seed)))
            continue
        ids += seed % 1000   # (ids need not begin at zero)
        if case.get("ids") == "sparse" and kind in ("i32", "i64"):  # odd multipliers: distinct ids stay distinct
            ids *= -7046029254386353131 if kind == "i64" else 2654435761
            if kind == "i32":
                ids = (ids << 32) >> 32
        vals = ids.to(torch.float64) * 0.25 if kind == "f64" else ids.to(DTYPES[kind])
        del ids
        cols.append(_column(vals, case.get("key_nulls", 0.0), rows, 2 * i + 1))
    return cols


def _value_columns(case, kinds, rows):
    # (the sum of squares of an integer column is a 64-bit integer: no variance of values that overflow it)
    squares = "var" in case.get("aggs", "") or "std" in case.get("aggs", "")
    cols = []
    for i, kind in enumerate(kinds):
        v = torch.empty(rows.n, dtype=DTYPES[kind], device="cuda")
        if kind in ("f32", "f64"):
            if case.get("skew") == "zipf":
                v.log_normal_(0.0, 1.0, generator=rows.gen)
            elif kind == "f32":
                v.uniform_(0.0, 1000.0, generator=rows.gen)
            else:
                v.normal_(0.0, 1.0, generator=rows.gen)
        else:
            span = {"i8": 100, "i16": 10_000, "i32": 1_000_000, "i64": 1_000_000_000}[kind]
            if squares:
                span = min(span, 10_000)
            v.random_(-span if kind == "i64" else 0, span, generator=rows.gen)
        nulls = case["nulls"] if case["do"] != "partition" or i == 0 else 0.0
        cols.append(_column(v, nulls, rows, 32 + i))
    return cols


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(1_000_003 * (seed + 1))
    n = case["rows"]
    if case["do"] == "partition":
        rows = _Rows(n, gen)
        keys = _key_columns(case, rows, seed)
        number = cb.Column.from_tensor(torch.arange(n, dtype=torch.int32, device="cuda"))
        return {"case": case, "table": cb.Table(keys + _value_columns(case, case["columns"].split(","), rows) + [number]),
                "nkeys": len(keys)}
    aggs = [Aggregation(KINDS[a]) for a in case["aggs"].split(",")]
    values = case["values"].split(",")
    if case["do"] == "stream":
        nkeys = len(case["keys"].split(","))
        tables = [_Rows(n, gen, b) for b in range(case["batches"])]
        batches = [cb.Table(_key_columns(case, t, seed) + _value_columns(case, values, t)) for t in tables]
        reqs = [cb.StreamingAggregationRequest(nkeys + i, a) for i in range(len(values)) for a in aggs]
        return {"case": case, "batches": batches, "nkeys": nkeys, "requests": reqs,
                "most": max(n, math.prod(_key_domains(case["keys"], case["groups"])))}
    rows = _Rows(n, gen)
    keys = cb.Table(_key_columns(case, rows, seed))
    vals = _value_columns(case, values, rows)
    return {"case": case, "keys": keys, "values": vals, "aggs": aggs,
            "policy": NullPolicy.INCLUDE if case["policy"] == "include" else NullPolicy.EXCLUDE,
            "filters": vals if case["dropna"] else []}


# ---------------------------------------------------------------------------------------------------- the calls
def run(state):
    case = state["case"]
    if case["do"] == "partition":
        table, offsets = hash_partition(state["table"], state["nkeys"], case["parts"])
        return InOrder(lambda: _ordered_partitions(table, offsets))
    if case["do"] == "stream":
        s = cb.StreamingGroupBy(list(range(state["nkeys"])), state["requests"], state["most"])
        for batch in state["batches"]:
            s.aggregate(batch)
        keys, results = s.finalize()
        return InOrder(lambda: _ordered_groups(keys, results))
    gb = cb.GroupBy(state["keys"], state["policy"], row_filters=state["filters"])
    keys, results = gb.aggregate([cb.GroupByRequest(v, state["aggs"]) for v in state["values"]])
    return InOrder(lambda: _ordered_groups(keys, results))


class InOrder(dict):
    """The columns of a result by name, brought into a defined row order when they are first read."""

    def __init__(self, columns):
        super().__init__()
        self._columns = columns

    def _read(self):
        if self._columns is not None:
            columns, self._columns = self._columns, None
            self.update(columns())

    def __iter__(self):
        self._read()
        return super().__iter__()

    def __len__(self):
        self._read()
        return super().__len__()

    def __getitem__(self, name):
        self._read()
        return super().__getitem__(name)

    def keys(self):
        self._read()
        return super().keys()

    def values(self):
        self._read()
        return super().values()

    def items(self):
        self._read()
        return super().items()


def _elements(col):
    """(elements of a fixed-width column with nulls as zero, validity or None)"""
    width = type_width(col.type_id)
    dtype = torch.from_numpy(np.zeros(1, STORAGE_DTYPE[col.type_id])).dtype
    if col.size == 0:
        return torch.zeros(0, dtype=dtype, device="cuda"), None
    v = col.data[:col.size * width].view(dtype)
    ok = _valid(col)
    return (v, None) if ok is None else (torch.where(ok, v, torch.zeros_like(v)), ok)


def _valid(col):
    if col.mask is None or col.size == 0:
        return None
    words = col.mask.view(torch.int32)[:(col.size + 31) // 32]
    shifts = torch.arange(32, dtype=torch.int32, device=words.device)
    return (((words.unsqueeze(1) >> shifts) & 1) != 0).view(-1)[:col.size]


def _offsets(col):
    return col.offsets.view(torch.int64 if col.offsets_type == TypeId.INT64 else torch.int32)[:col.size + 1].to(torch.int64)


def _mix(h, x):
    h = h * -7046029254386353131 + (x + 1) * -4417276706812531889
    return h ^ ((h >> 29) & 0x7FFFFFFFF)


def _string_hashes(col):
    offs = _offsets(col)
    lens = offs[1:] - offs[:-1]
    at = torch.arange(int(offs[-1]), device=offs.device) - torch.repeat_interleave(offs[:-1], lens)
    powers = torch.tensor([pow(0x9E3779B97F4A7C15, i + 1, 1 << 64) for i in range(int(lens.max()) if lens.numel() else 0)],
                          dtype=torch.uint64).view(torch.int64).to(offs.device)
    sums = torch.zeros(at.numel() + 1, dtype=torch.int64, device=offs.device)
    torch.cumsum((col.data[:at.numel()].to(torch.int64) + 1) * powers[at], 0, out=sums[1:])
    return sums[offs[1:]] - sums[offs[:-1]]


def _rank_of_keys(keys):
    """A permutation that orders the groups by their keys: by value for one integer column, else by a 64-bit mix."""
    if len(keys) == 1 and keys[0].mask is None and keys[0].type_id != TypeId.STRING:
        return torch.argsort(_elements(keys[0])[0])
    h = None
    for c in keys:
        if c.type_id == TypeId.STRING:
            x = _string_hashes(c)
        else:
            x, ok = _elements(c)
            x = x.view(torch.int64) if x.dtype == torch.float64 else x.to(torch.int64)
            if ok is not None:
                x = torch.where(ok, x, torch.full_like(x, -8446744073709551557))
        h = _mix(torch.zeros_like(x) if h is None else h, x)
    return torch.argsort(h)


def _put(out, name, col, order):
    if col.type_id == TypeId.STRING:
        offs = _offsets(col)
        lens = (offs[1:] - offs[:-1])[order]
        new = torch.zeros(col.size + 1, dtype=torch.int64, device=offs.device)
        torch.cumsum(lens, 0, out=new[1:])
        src = torch.repeat_interleave(offs[:-1][order] - new[:-1], lens) + torch.arange(int(new[-1]), device=offs.device)
        out[name + ".chars"], out[name + ".offsets"] = col.data[src], new
        return
    v, ok = _elements(col)
    out[name] = v[order]
    if ok is not None:
        out[name + ".valid"] = ok[order]


def _ordered_groups(keys, results):
    order = _rank_of_keys(keys.columns())
    out = {}
    for i, c in enumerate(keys.columns()):
        _put(out, "key%d" % i, c, order)
    for r, t in enumerate(results):
        for i, c in enumerate(t.columns()):
            _put(out, "result%d.%d" % (r, i), c, order)
    return out


def _ordered_partitions(table, offsets):
    cols = table.columns()
    starts = torch.tensor(offsets, dtype=torch.int64, device="cuda")
    row = _elements(cols[-1])[0].to(torch.int64)
    part = torch.searchsorted(starts, torch.arange(row.numel(), device="cuda"), right=True) - 1
    order = torch.argsort((part << 32) | row)
    out = {"offsets": np.asarray(offsets, dtype=np.int64)}
    for i, c in enumerate(cols):
        _put(out, "column%d" % i, c, order)
    return out


# ---------------------------------------------------------------------------------------------------- what it needs
def _distinct(n, groups, skew):
    """Expected number of groups among n rows."""
    if skew == "uniform":
        return groups * -math.expm1(n * math.log1p(-1.0 / groups)) if groups > 1 else 1.0
    p = np.arange(1, groups + 1, dtype=np.float64) ** -1.1
    p /= p.sum()
    return float(-np.expm1(n * np.log1p(-p[1:])).sum()) + 1.0


def _row_bytes(kinds):
    return sum(MEAN_STRING + 4 if k == "str" else type_width(TYPE_IDS[k]) for k in kinds)


def work(case):
    n, keys = case["rows"], case["keys"].split(",")
    if case["do"] == "partition":
        cols = case["columns"].split(",")
        table = n * (_row_bytes(keys + cols) + 4) + (n / 8 if case["nulls"] else 0)
        return {"bytes": 2.0 * table, "flops": float(n * len(keys))}
    vals, aggs = case["values"].split(","), case["aggs"].split(",")
    n *= case.get("batches", 1)
    masks = len(vals) * (case["nulls"] > 0) + len(keys) * (case.get("key_nulls", 0.0) > 0)
    groups = _distinct(n, math.prod(_key_domains(case["keys"], case["groups"])), case.get("skew", "uniform"))
    outs = sum(type_width(result_type(TYPE_IDS[v], KINDS[a])) for v in vals for a in aggs)
    return {"bytes": n * (_row_bytes(keys + vals) + masks / 8.0) + groups * (_row_bytes(keys) + outs),
            "flops": float(n * len(vals) * len(aggs))}


def tolerance(case):
    """Keys, counts, integer results and moved rows are exact; sums, means and variances of floats depend on the order of
    the additions: a few roundings of the source type for each of them."""
    if case["do"] == "partition":
        return "exact"
    if "f32" in case["values"]:
        return {"rel": 1e-5}
    if "std" in case["aggs"]:   # the root of a difference of nearly equal sums, where a group's values lie close together
        return {"rel": 1e-12, "max": 1e-8}
    if "f64" in case["values"] or "mean" in case["aggs"] or "var" in case["aggs"] or "std" in case["aggs"]:
        return {"rel": 1e-12}
    return "exact"
