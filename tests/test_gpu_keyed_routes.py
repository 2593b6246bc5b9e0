"""Which calls over keys that do not pack are served by k_keyed (the statistics of a call tell: its dictionary has the smallest power of
two of 1.5 cells per row that there can be), and what comes of those that it gives up or that are handed on."""
import ctypes as C

import numpy as np
import pytest
import torch

import cudf_b200 as cb
from cudf_b200 import _lib
from cudf_b200.column import TorchAllocator
from cudf_b200.groupby import _adopt_result, _check, _requests_to_c
from cudf_b200.types import TypeId

pytestmark = pytest.mark.gpu
SHAPES = ["str", "str,i16", "long", "f64", "i64,i32"]


def _strings(ids, words, large=False, front=0):
    """Every id as a string of `words` times its 8 bytes; `front`: a column sliced behind so many other rows."""
    ids = torch.cat([torch.full((front,), -7, dtype=torch.int64, device="cuda"), ids]) if front else ids
    chars = ids.view(-1, 1).repeat(1, words).view(-1).view(torch.uint8)
    offsets = torch.arange(ids.numel() + 1, dtype=torch.int64 if large else torch.int32, device="cuda") * 8 * words
    return cb.Column(TypeId.STRING, ids.numel() - front, chars, None, front, 0, offsets.view(torch.uint8), TypeId.INT64 if large else TypeId.INT32)


def _keys(shape, ids, **how):
    if shape == "f64":
        return [cb.Column.from_tensor(ids.to(torch.float64) * 0.5)]
    if shape == "i64,i32":
        return [cb.Column.from_tensor(ids * 1_000_003), cb.Column.from_tensor((ids % 7).to(torch.int32))]
    s = _strings(ids, 5 if shape == "long" else 1, **how)
    return [s, cb.Column.from_tensor((ids % 9).to(torch.int16))] if shape == "str,i16" else [s]


def _ids_of(shape, keys):
    k = keys.columns()[0]
    if shape == "f64":
        return (k.data[:8 * k.size].view(torch.float64) * 2).to(torch.int64)
    if shape == "i64,i32":
        return k.data[:8 * k.size].view(torch.int64) // 1_000_003
    words = 5 if shape == "long" else 1
    offsets = k.offsets.view(torch.int64 if k.offsets_type == TypeId.INT64 else torch.int32)[:k.size + 1]
    assert torch.equal(offsets.to(torch.int64), torch.arange(k.size + 1, device="cuda") * 8 * words)
    return k.data[:8 * words * k.size].view(torch.int64).view(-1, words)[:, -1]


def _requests(v):
    return [cb.GroupByRequest(cb.Column.from_tensor(v), [cb.aggregation.sum(), cb.aggregation.max(), cb.aggregation.count()])]


def _inputs(n, groups, seed=1):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    ids = torch.randint(0, groups, (n,), device="cuda", generator=gen)
    ids[:min(n, groups)] = torch.arange(min(n, groups), device="cuda")
    return ids, torch.randint(-10**9, 10**9, (n,), device="cuda", generator=gen)


def _compare(shape, ids, v, got):
    keys, (res,) = got
    at, order = torch.sort(_ids_of(shape, keys))
    uniq, where, counts = torch.unique(ids, return_inverse=True, return_counts=True)
    assert torch.equal(at, uniq)
    if shape == "i64,i32":
        assert torch.equal(keys.columns()[1].data[:4 * at.numel()].view(torch.int32)[order].to(torch.int64), uniq % 7)
    if shape == "str,i16":
        assert torch.equal(keys.columns()[1].data[:2 * at.numel()].view(torch.int16)[order].to(torch.int64), uniq % 9)
    g = at.numel()
    sums, most, count = (c.data for c in res.columns())
    assert torch.equal(sums[:8 * g].view(torch.int64)[order], torch.zeros_like(uniq).index_add_(0, where, v))
    assert torch.equal(most[:8 * g].view(torch.int64)[order], torch.full_like(uniq, -10**10).scatter_reduce_(0, where, v, "amax"))
    assert torch.equal(count[:4 * g].view(torch.int32)[order].to(torch.int64), counts)


def _cells(rows):
    cap = 1024
    while cap < 1.5 * rows and cap < 1 << 22:
        cap *= 2
    return cap


def _served(st, cells):
    return st.table_attempts == 1 and st.used_shared_table and st.table_capacity in cells


@pytest.mark.parametrize("variant", [0, 9])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("n,groups", [(1, 1), (33, 5), (4097, 40), (90_001, 60_000), (700_003, 3000)])
def test_served(n, groups, shape, variant):
    ids, v = _inputs(n, groups)
    _compare(shape, ids, v, cb.GroupBy(cb.Table(_keys(shape, ids)), table_variant=variant).aggregate(_requests(v)))
    assert _served(cb.last_call_stats(), [_cells(n)])


@pytest.mark.parametrize("large,front", [(True, 0), (False, 3), (True, 37)])
@pytest.mark.parametrize("shape", ["str", "str,i16", "long"])
def test_served_offsets_of_both_widths_and_slices(shape, large, front):
    ids, v = _inputs(90_001, 5000)
    _compare(shape, ids, v, cb.GroupBy(cb.Table(_keys(shape, ids, large=large, front=front))).aggregate(_requests(v)))
    assert _served(cb.last_call_stats(), [_cells(90_001)])


@pytest.mark.parametrize("shape", ["str", "i64,i32"])
def test_served_behind_a_sample(shape):
    """More rows than a dictionary has ids."""
    ids, v = _inputs(3_200_003, 100_000)
    _compare(shape, ids, v, cb.GroupBy(cb.Table(_keys(shape, ids))).aggregate(_requests(v)))
    assert _served(cb.last_call_stats(), [1 << 22])


@pytest.mark.parametrize("variant", [0, 9])
@pytest.mark.parametrize("shape", SHAPES)
def test_more_keys_than_cells(shape, variant):
    """A hint far too low lets the attempt begin: the dictionary runs full with ids handed out, cells claimed and never published, and
    rows waiting for them.  The call goes on as without it."""
    ids, v = _inputs(3_500_000, 3_500_000)
    _compare(shape, ids, v, cb.GroupBy(cb.Table(_keys(shape, ids)), expected_groups=1000, table_variant=variant).aggregate(_requests(v)))
    assert not _served(cb.last_call_stats(), [1 << 14])


def _milliseconds(gb, reqs):
    times = []
    for _ in range(8):
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        gb.aggregate(reqs)
        t1.record()
        torch.cuda.synchronize()
        times.append(t0.elapsed_time(t1))
    return times


@pytest.mark.parametrize("shape", ["str", "i64,i32"])
def test_a_frequent_key_among_many(shape):
    """Half of the rows have one key, which is met after hundreds of others: it is aggregated in shared memory all the same.  (As
    reductions of one global word per cell its million rows take several milliseconds, the call less than half a one.)"""
    n, groups = 1_900_000, 200_000
    ids, _ = _inputs(n, groups)
    ids[torch.rand(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(8)) < 0.5] = 77_777
    v = torch.arange(n, device="cuda") % 1000
    reqs = [r for c in range(5) for r in _requests(v + c)]
    times = _milliseconds(cb.GroupBy(cb.Table(_keys(shape, ids))), reqs)
    assert _served(cb.last_call_stats(), [1 << 22])
    assert sorted(times)[len(times) // 2] < 1.5, times
    _compare(shape, ids, v, cb.GroupBy(cb.Table(_keys(shape, ids))).aggregate(_requests(v)))


def test_skewed_keys_of_which_a_sample_says_too_few():
    """Zipf-distributed keys: 2048 rows tell a tenth of the groups.  The dictionary holds them all the same."""
    n = 3_200_003
    weights = torch.cumsum(torch.arange(1, 1_000_001, device="cuda", dtype=torch.float64) ** -1.1, 0)
    ids = torch.searchsorted(weights, torch.rand(n, device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(9)) * weights[-1])
    v = torch.arange(n, device="cuda") % 1000
    _compare("i64,i32", ids, v, cb.GroupBy(cb.Table(_keys("i64,i32", ids))).aggregate(_requests(v)))
    assert _served(cb.last_call_stats(), [1 << 22])


# few groups, groups in runs, cells by rows: what dictionary ids serve better than sums of doubles as compare-and-swap loops
@pytest.mark.parametrize("shape,n,groups,runs,columns,served", [
    ("str", 2_200_000, 2, False, 1, False), ("str", 2_200_000, 2, False, 0, True), ("str", 2_200_000, 400, False, 1, True), ("str", 2_200_000, 400, True, 1, False),
    ("str", 2_200_000, 400, True, 0, True), ("str", 6_400_000, 400, False, 5, False), ("i64,i32", 4_400_000, 400, False, 1, True), ("i64,i32", 4_400_000, 400, True, 1, False),
    ("i64,i32", 4_400_000, 4, True, 1, True), ("i64,i32", 6_400_000, 400, False, 5, False)])
def test_where_ids_serve_a_call_too(shape, n, groups, runs, columns, served):
    ids, v = _inputs(n, groups)
    ids = ids.sort().values if runs else ids
    reqs = _requests(v) + [cb.GroupByRequest(cb.Column.from_tensor(v.to(torch.float64) + c), [cb.aggregation.sum(), cb.aggregation.count()]) for c in range(columns)]
    keys, res = cb.GroupBy(cb.Table(_keys(shape, ids))).aggregate(reqs)
    assert _served(cb.last_call_stats(), [_cells(n)]) == served
    _compare(shape, ids, v, (keys, res[:1]))


@pytest.mark.parametrize("groups,ids_pay", [(10, False), (900, True), (20_000, True)])
def test_ids_by_the_sample_beyond_its_rows(groups, ids_pay):
    """More than 16M rows: row keys where the cache of their pass holds the groups, else ids, behind which a table is sized by their
    number."""
    ids, v = _inputs((1 << 24) + 5, groups)
    _compare("i64,i32", ids, v, cb.GroupBy(cb.Table(_keys("i64,i32", ids))).aggregate(_requests(v)))
    st = cb.last_call_stats()
    assert (st.used_shared_table and st.table_capacity == 1 << 18) != ids_pay   # (2^18 slots: row keys; ids may go through partitions)


class Refuses(TorchAllocator):
    """Has no memory for the first `times` result buffers."""

    def __init__(self, times):
        super().__init__("cuda")
        self.times = times

    def _alloc(self, nbytes, stream, ctx):
        self.times -= 1
        return None if self.times >= 0 else super()._alloc(nbytes, stream, ctx)


@pytest.mark.parametrize("shape", ["str", "i64,i32"])
def test_results_that_do_not_fit_beside_the_dictionary(shape):
    n = 500_003
    ids, v = _inputs(n, 1000)
    gb, reqs, alloc = cb.GroupBy(cb.Table(_keys(shape, ids))), _requests(v), Refuses(1)
    keep, res = [], _lib.GroupbyResult()
    _check(_lib.load().b2_groupby_aggregate(gb._handle, _requests_to_c(reqs, keep), len(reqs), C.c_void_p(torch.cuda.current_stream().cuda_stream),
                                            C.byref(alloc.struct), C.byref(res)))
    _compare(shape, ids, v, _adopt_result(res, alloc))
    assert alloc.times < 0 and not alloc.live and not _served(cb.last_call_stats(), [_cells(n)])


def test_one_sample_of_the_rows_is_enough():
    """More groups than a dictionary takes: k_keyed hands its sample on, and the call ends with row keys, as it does where no sample is
    taken (table_variant 7)."""
    n = (1 << 22) + 5
    ids, v = _inputs(n, n)
    launches = []
    for variant in (7, 0):
        keys, _ = cb.GroupBy(cb.Table(_keys("i64,i32", ids)), table_variant=variant).aggregate(_requests(v))
        assert keys.num_rows() == n
        launches.append(cb.last_call_stats().kernel_launches)
    assert launches[1] == launches[0] + 1


@pytest.mark.parametrize("shape", ["str", "str,i16"])
def test_counts_of_a_float_column_are_no_sums(shape):
    n, groups = 2_200_003, 5000
    ids, v = _inputs(n, groups)
    keys, (res,) = cb.GroupBy(cb.Table(_keys(shape, ids))).aggregate([cb.GroupByRequest(cb.Column.from_tensor(v.to(torch.float64)), [cb.aggregation.count()])])
    assert _served(cb.last_call_stats(), [_cells(n)])
    at, order = torch.sort(_ids_of(shape, keys))
    assert torch.equal(at, torch.arange(groups, device="cuda"))
    assert torch.equal(res.columns()[0].data[:4 * groups].view(torch.int32)[order].to(torch.int64), torch.bincount(ids, minlength=groups))
