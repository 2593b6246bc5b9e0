"""`expected_groups` beside the rule that sends rows to the partitions: a call that is told its groups decides before it allocates,
and one whose table holds as many groups as there are rows is never turned away from it."""
import numpy as np
import pytest

import cudf_b200 as cb
from cudf_b200.types import HostColumn, Kind, TypeId
from tests.test_gpu_comm import _multi, comm  # noqa: F401  (a fixture)
from tests.test_gpu_parity import check

pytestmark = pytest.mark.gpu
FOUR = [Kind.SUM, Kind.MIN, Kind.MAX, Kind.COUNT_VALID]


def _distinct(n):
    rng = np.random.default_rng(n)
    return HostColumn.from_numpy(rng.permutation(n).astype(np.int64)), HostColumn.from_numpy(rng.integers(-10**9, 10**9, n))


# dense ids in a table at full capacity, above the limit that a sample would be held against: at its lower end, inside, and
# where the hint alone decides for partitions
@pytest.mark.parametrize("n,aggs", [(340_000, FOUR), (450_000, FOUR), (523_000, FOUR), (561_000, FOUR),
                                    (495_000, [Kind.SUM]), (600_000, [Kind.SUM]), (600_000, [Kind.MEAN]), (755_000, [Kind.SUM]), (810_000, [Kind.SUM])])
@pytest.mark.parametrize("share", [1.0, 0.85])
def test_nearly_every_row_a_group(n, aggs, share):
    k, v = _distinct(n)
    check([k], [(v, aggs)], expected_groups=int(n * share))
    assert cb.last_call_stats().table_attempts == 1


@pytest.mark.parametrize("n,aggs", [(450_000, FOUR), (600_000, [Kind.SUM])])
def test_nearly_every_row_a_group_on_a_communicator(comm, monkeypatch, n, aggs):  # noqa: F811
    import functools
    from cudf_b200 import groupby
    k, v = _distinct(n)
    monkeypatch.setattr(groupby, "GroupBy", functools.partial(groupby.GroupBy, expected_groups=n))
    keys, res = _multi(comm, [k], [(v, aggs)])
    order = np.argsort(keys[0].values())
    assert np.array_equal(keys[0].values()[order], np.arange(n))
    assert np.array_equal(res[0][0].values()[order], v.values()[np.argsort(k.values())])


# 2.5M rows, four accumulators: a sample of dense ids says partitions from 25K groups on, a hint from 69K on
@pytest.mark.parametrize("groups,hint,partitioned", [(60_000, 60_000, False), (60_000, 200_000, True), (100_000, 100_000, True)])
def test_a_hinted_call_allocates_one_table_or_none(groups, hint, partitioned):
    n = 2_500_000
    rng = np.random.default_rng(groups)
    k = HostColumn.from_numpy(rng.integers(0, groups, n))
    check([k], [(HostColumn.from_numpy(rng.integers(-10**9, 10**9, n)), FOUR)], expected_groups=hint)
    st = cb.last_call_stats()
    assert st.table_attempts == 1 and st.used_shared_table != partitioned


def _zipf(rng, n, groups):
    return np.searchsorted(np.cumsum(np.arange(1, groups + 1) ** -1.1) / np.sum(np.arange(1, groups + 1) ** -1.1), rng.random(n))


# 2.5M rows, four accumulators, hints beyond the line: what a sample of the rows says against them
@pytest.mark.parametrize("keys,hint,partitioned", [("sparse", 80_000, True), ("far more", 80_000, True), ("compact", 80_000, False), ("skewed", 80_000, False),
                                                   ("far fewer", 80_000, False)])
def test_a_hint_is_held_against_a_sample(keys, hint, partitioned):
    n = 2_500_000
    rng = np.random.default_rng(hint)
    k = {"sparse": lambda: rng.integers(0, 100_000, n) * 7046029254386353131, "far more": lambda: rng.integers(0, 400_000, n) * 7046029254386353131,
         "compact": lambda: rng.integers(0, 2000, n), "skewed": lambda: _zipf(rng, n, 80_000) * 7046029254386353131,
         "far fewer": lambda: rng.integers(0, 20_000, n) * 7046029254386353131}[keys]()
    check([HostColumn.from_numpy(k.astype(np.int64))], [(HostColumn.from_numpy(rng.integers(-10**9, 10**9, n)), FOUR)], expected_groups=hint)
    st = cb.last_call_stats()
    assert st.table_attempts == 1 and st.used_shared_table != partitioned


@pytest.mark.parametrize("runs", [False, True])
def test_ids_of_few_rows_stay_in_a_table(runs):
    """Dictionary ids, their number known: with 2.5M rows partitions start later than with 16M, and a sample of rows in runs, of which no
    two have the same key, says nothing against it."""
    import torch
    n, groups = 2_500_000, 14_000
    ids = torch.randint(0, groups, (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    ids = ids.sort().values if runs else ids
    offsets = torch.arange(n + 1, dtype=torch.int32, device="cuda") * 8
    key = cb.Column(TypeId.STRING, n, ids.view(torch.uint8), None, 0, 0, offsets.view(torch.uint8), TypeId.INT32)
    v = torch.rand(n, dtype=torch.float64, device="cuda")
    keys, (res,) = cb.GroupBy(cb.Table([key])).aggregate([cb.GroupByRequest(cb.Column.from_tensor(v), [cb.aggregation.count(), cb.aggregation.sum(), cb.aggregation.variance()])])
    st = cb.last_call_stats()
    assert st.table_attempts == 1 and st.used_shared_table
    at, order = keys.columns()[0].data[:8 * groups].view(torch.int64).sort()
    assert torch.equal(at, torch.arange(groups, device="cuda"))
    assert torch.equal(res.columns()[0].data[:4 * groups].view(torch.int32)[order].to(torch.int64), torch.bincount(ids, minlength=groups))
    exact = torch.zeros(groups, dtype=torch.float64, device="cuda").index_add_(0, ids, v)
    assert torch.allclose(res.columns()[1].data[:8 * groups].view(torch.float64)[order], exact, rtol=1e-12, atol=0)


@pytest.mark.parametrize("aggs,partitioned", [([cb.aggregation.sum(), cb.aggregation.max()], False), ([cb.aggregation.count()], True)])
def test_rows_in_runs_of_one_key(aggs, partitioned):
    """Rows in key order visit a table's lines in order: 8 bytes of values a row are not moved to partitions, counts are."""
    import torch
    n, groups = (1 << 23) + 77, 60_000
    ids = torch.randint(0, groups, (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).sort().values
    v = torch.randint(-10**9, 10**9, (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
    keys, (res,) = cb.GroupBy(cb.Table([cb.Column.from_tensor(ids)]), expected_groups=groups).aggregate([cb.GroupByRequest(cb.Column.from_tensor(v), aggs)])
    st = cb.last_call_stats()
    assert st.table_attempts == 1 and st.used_shared_table != partitioned
    at, order = keys.columns()[0].data[:8 * groups].view(torch.int64).sort()
    assert torch.equal(at, torch.arange(groups, device="cuda"))
    first = res.columns()[0].data
    if partitioned:
        assert torch.equal(first[:4 * groups].view(torch.int32)[order].to(torch.int64), torch.bincount(ids, minlength=groups))
    else:
        assert torch.equal(first[:8 * groups].view(torch.int64)[order], torch.zeros(groups, dtype=torch.int64, device="cuda").index_add_(0, ids, v))


def test_groups_that_chunks_hold_stay_in_a_table(comm):  # noqa: F811
    """A communicator of one rank exchanges up to 16384 groups in chunks, without reading its table back; a list from partitions would
    take a second exchange."""
    n, groups = 8_000_000, 11_000
    rng = np.random.default_rng(2)
    k = rng.integers(0, groups, n)
    v = rng.integers(-1000, 1000, n)
    keys, res = _multi(comm, [HostColumn.from_numpy(k)], [(HostColumn.from_numpy(v), FOUR)])
    assert cb.last_call_stats().table_attempts == 1
    order = np.argsort(keys[0].values())
    assert np.array_equal(keys[0].values()[order], np.arange(groups))
    assert np.array_equal(res[0][3].values()[order], np.bincount(k, minlength=groups))
    assert np.array_equal(res[0][0].values()[order], np.bincount(k, weights=v, minlength=groups).astype(np.int64))


# 2.5M rows: a hint far too low, and rows in runs of one key, of which a sample sees none twice
@pytest.mark.parametrize("runs,groups,hint,floats,partitioned", [(False, 400_000, 8000, False, True), (True, 30_000, 30_000, False, True), (True, 30_000, 30_000, True, False)])
def test_a_sample_that_tells_far_more_than_the_hint(runs, groups, hint, floats, partitioned):
    n = 2_500_000
    rng = np.random.default_rng(groups)
    k = rng.integers(0, groups, n)
    k = np.sort(k) if runs else k * 7046029254386353131
    v = rng.integers(-10**6, 10**6, n)
    check([HostColumn.from_numpy(k)], [(HostColumn.from_numpy(v.astype(np.float64) if floats else v), [Kind.SUM, Kind.MAX] if floats else FOUR)], expected_groups=hint)
    st = cb.last_call_stats()
    assert (st.table_attempts == 2 and st.table_capacity != 2 * hint + 64) == partitioned
    assert partitioned or (st.table_attempts == 1 and st.table_capacity == 2 * hint + 64)
