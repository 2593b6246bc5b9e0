"""Results of the partitioned path written straight into columns that were allocated for the whole key box: calls whose columns do
not fit memory, and columns that are copied because the box has many more positions than groups."""
import ctypes as C

import pytest
import torch

import cudf_b200 as cb
from cudf_b200 import _lib
from cudf_b200.column import TorchAllocator
from cudf_b200.groupby import _adopt_result, _check, _requests_to_c

pytestmark = pytest.mark.gpu
MB = 1 << 20


class Bounded(TorchAllocator):
    """Refuses a result buffer of more than `most` bytes."""

    def __init__(self, device, most):
        super().__init__(device)
        self.most, self.refused = most, 0

    def _alloc(self, nbytes, stream, ctx):
        if nbytes > self.most:
            self.refused += 1
            return None
        return super()._alloc(nbytes, stream, ctx)


def _aggregate(gb, requests, alloc):
    keep, res = [], _lib.GroupbyResult()
    _check(_lib.load().b2_groupby_aggregate(gb._handle, _requests_to_c(requests, keep), len(requests),
                                            C.c_void_p(torch.cuda.current_stream().cuda_stream), C.byref(alloc.struct), C.byref(res)))
    return _adopt_result(res, alloc)


@pytest.mark.parametrize("groups,hint", [(50_000, 200_000), (150_000, 0), (150_000, 150_000)])
def test_columns_for_the_whole_box_do_not_fit(groups, hint):
    n, box = 5_000_003, 1_200_000        # (a position for every four rows: the results go straight into the columns)
    gen = torch.Generator(device="cuda").manual_seed(groups)
    at = torch.randperm(box, device="cuda", generator=gen)[:groups].sort().values
    at[0], at[-1] = 0, box - 1
    ids = torch.randint(0, groups, (n,), device="cuda", generator=gen)
    ids[:groups] = torch.arange(groups, device="cuda")
    v = torch.randint(-1000, 1000, (n,), device="cuda", generator=gen)
    gb = cb.GroupBy(cb.Table([cb.Column.from_tensor(at[ids])]), expected_groups=hint)
    reqs = [cb.GroupByRequest(cb.Column.from_tensor(v), [cb.aggregation.sum(), cb.aggregation.max(), cb.aggregation.count()])]
    sums = torch.zeros(groups, dtype=torch.int64, device="cuda").index_add_(0, ids, v)
    most = torch.full((groups,), -10**6, dtype=torch.int64, device="cuda").scatter_reduce_(0, ids, v, "amax")
    for limit in (64 * MB, 4 * MB):      # a column of the box has 9.6 MB, one of the groups at most 1.2
        alloc = Bounded("cuda", limit)
        keys, (res,) = _aggregate(gb, reqs, alloc)
        assert (alloc.refused > 0) == (limit == 4 * MB) and not alloc.live
        assert keys.num_rows() == groups
        k = keys.columns()[0].data[:groups * 8].view(torch.int64)
        order = torch.argsort(k)
        assert torch.equal(k[order], at)
        got = [c.data for c in res.columns()]
        assert torch.equal(got[0][:groups * 8].view(torch.int64)[order], sums)
        assert torch.equal(got[1][:groups * 8].view(torch.int64)[order], most)
        assert torch.equal(got[2][:groups * 4].view(torch.int32)[order].to(torch.int64), torch.bincount(ids, minlength=groups))


@pytest.fixture(scope="module")
def sparse_box():
    """160M rows over 13.3M ids in a box of 40M positions."""
    n, groups = 160_000_000, 13_300_000
    gen = torch.Generator(device="cuda").manual_seed(1)
    ids = torch.randint(0, groups, (n,), device="cuda", generator=gen, dtype=torch.int32)
    ids[:groups] = torch.arange(groups, device="cuda", dtype=torch.int32)
    v = torch.randint(-1000, 1000, (n,), device="cuda", generator=gen, dtype=torch.int32)
    gb = cb.GroupBy(cb.Table([cb.Column.from_tensor(ids * 3)]), expected_groups=groups)
    aggs = [cb.aggregation.sum(), cb.aggregation.mean(), cb.aggregation.sum_of_squares(), cb.aggregation.variance(), cb.aggregation.std()]
    expected = torch.zeros(groups, dtype=torch.int64, device="cuda")
    for lo in range(0, n, 40_000_000):
        expected.index_add_(0, ids[lo:lo + 40_000_000], v[lo:lo + 40_000_000].to(torch.int64))
    return gb, [cb.GroupByRequest(cb.Column.from_tensor(v), aggs)], groups, expected


def _check_sums(keys, res, groups, expected):
    assert keys.num_rows() == groups
    at = keys.columns()[0].data[:groups * 4].view(torch.int32).to(torch.int64) // 3
    assert torch.equal(torch.zeros_like(expected).scatter_(0, at, res.columns()[0].data[:groups * 8].view(torch.int64)), expected)


def test_copied_columns_are_written_when_the_call_returns(sparse_box):
    gb, reqs, groups, expected = sparse_box
    other = torch.cuda.Stream()
    for _ in range(3):
        torch.cuda.synchronize()
        held = torch.cuda.memory_allocated()
        keys, (res,) = gb.aggregate(reqs)
        assert torch.cuda.memory_allocated() - held < 7 * groups * 8   # (copied: a column of the box has 160 or 320 MB)
        with torch.cuda.stream(other):   # (no wait for the stream of the call)
            seen = [c.data.clone() for c in reversed(res.columns())]
        torch.cuda.synchronize()
        for a, c in zip(seen, reversed(res.columns())):
            assert torch.equal(a, c.data)
        _check_sums(keys, res, groups, expected)
        del keys, res, seen


def test_a_column_is_kept_where_its_copy_finds_no_memory(sparse_box):
    gb, reqs, groups, expected = sparse_box

    class Full(TorchAllocator):          # no memory for the copies of columns, which have 53 or 106 MB
        def _alloc(self, nbytes, stream, ctx):
            return None if 50_000_000 < nbytes < 110_000_000 else super()._alloc(nbytes, stream, ctx)

    alloc = Full("cuda")
    keys, (res,) = _aggregate(gb, reqs, alloc)
    assert res.columns()[0].data.untyped_storage().nbytes() > 300_000_000 and not alloc.live
    _check_sums(keys, res, groups, expected)
