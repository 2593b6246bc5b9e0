"""Sums of one FLOAT64 column over keys that do not pack, from the row counts on from which dictionary ids bring them to exact cells:
they are not left to a pass that adds doubles one after the other."""
import numpy as np
import pytest
import torch

import cudf_b200 as cb
from cudf_b200.types import TypeId

pytestmark = pytest.mark.gpu


def _strings(ids):
    """One-byte strings."""
    n = ids.numel()
    offsets = torch.arange(n + 1, dtype=torch.int32, device="cuda")
    return cb.Column(TypeId.STRING, n, (ids + 97).to(torch.uint8), None, 0, 0, offsets.view(torch.uint8), TypeId.INT32)


def _sums(keys, v):
    kt, (r,) = cb.GroupBy(cb.Table(keys)).aggregate([cb.GroupByRequest(cb.Column.from_tensor(v), [cb.aggregation.sum(), cb.aggregation.mean(), cb.aggregation.count()])])
    return [c.to_host().values() for c in r.columns()]


@pytest.mark.parametrize("beside", [False, True])
def test_strings(beside):
    """8M times 0.1 in two groups.  A CTA rounds its part of a group's sum once per 1024 addends and at the merge: 4096 + 296 half units
    of the sum, 5e-13 if all went one way, 7e-15 as their root.  Every addend rounded (the same way each, for they are equal)
    gives about an eighth of a unit per row of a CTA and group, 14000 rows here: 2e-13."""
    n = (1 << 23) + 3
    ids = torch.randint(0, 2, (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
    keys = [_strings(ids)] + ([cb.Column.from_tensor((ids * 0).to(torch.int8))] if beside else [])
    for _ in range(2):
        s, m, c = _sums(keys, torch.full((n,), 0.1, dtype=torch.float64, device="cuda"))
        assert sorted(c) == sorted(torch.bincount(ids).tolist())
        assert np.all(np.abs(s - 0.1 * c) <= 3e-14 * 0.1 * c) and np.all(np.abs(m - 0.1) <= 3e-14 * 0.1)


@pytest.mark.parametrize("floats", [False, True])
def test_wide_keys(floats):
    """A FLOAT64 key and a composite of 96 bits, 2000 groups: the table behind the ids is sized by their number."""
    n, groups = (1 << 22) + 5, 2000
    ids = torch.randint(0, groups, (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    ids[:groups] = torch.arange(groups, device="cuda")
    keys = [cb.Column.from_tensor(ids.to(torch.float64) * 0.5)] if floats else [cb.Column.from_tensor(ids * 1_000_003), cb.Column.from_tensor((ids % 7).to(torch.int32))]
    v = torch.rand(n, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(6))
    s, m, c = _sums(keys, v)
    assert cb.last_call_stats().table_capacity == 2 * groups + 64
    assert s.size == groups and sorted(c) == sorted(torch.bincount(ids).tolist())
    exact = torch.zeros(groups, dtype=torch.float64, device="cuda").index_add_(0, ids, v).sort().values.cpu().numpy()
    assert np.allclose(np.sort(s), exact, rtol=1e-12, atol=0) and np.allclose(m, s / c, rtol=1e-15, atol=0)


@pytest.mark.parametrize("hint", [100, 400_000])
def test_a_hint_that_is_off(hint):
    """Whether ids serve the call is for the sample to say, as it is without a hint; the dictionary of a pass that adds doubles would have 2^11 or
    2^22 cells."""
    n, groups = (1 << 22) + 5, 2000
    ids = torch.randint(0, groups, (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    ids[:groups] = torch.arange(groups, device="cuda")
    v = torch.rand(n, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(6))
    gb = cb.GroupBy(cb.Table([cb.Column.from_tensor(ids.to(torch.float64) * 0.5)]), expected_groups=hint)
    _, (r,) = gb.aggregate([cb.GroupByRequest(cb.Column.from_tensor(v), [cb.aggregation.sum(), cb.aggregation.count()])])
    assert cb.last_call_stats().table_capacity not in (1 << 11, 1 << 22)
    s, c = [x.to_host().values() for x in r.columns()]
    exact = torch.zeros(groups, dtype=torch.float64, device="cuda").index_add_(0, ids, v).sort().values.cpu().numpy()
    assert np.allclose(np.sort(s), exact, rtol=1e-12, atol=0) and sorted(c) == sorted(torch.bincount(ids).tolist())
