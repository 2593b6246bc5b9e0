"""Packed keys whose table of the first attempt does not hold the groups, around the rows from which on they are partitioned, and
inputs that the sample sends there at once: against the oracle."""
import numpy as np
import pytest

import cudf_b200 as cb
from cudf_b200.types import HostColumn, Kind, NullPolicy
from tests.test_gpu_parity import check

pytestmark = pytest.mark.gpu
INT = [Kind.SUM, Kind.MIN, Kind.MAX, Kind.COUNT_VALID]


@pytest.mark.parametrize("n,groups", [(262_143, 110_000), (262_144, 110_000), (524_287, 300_000), (524_288, 300_000), (2_500_000, 60_000)])
@pytest.mark.parametrize("sparse", [False, True])
def test_rows_and_groups(n, groups, sparse):
    rng = np.random.default_rng(n + groups)
    g = rng.integers(0, groups, n)
    k = g * 7046029254386353131 if sparse else g + 17
    key = HostColumn.from_numpy(k.astype(np.int64), valid=rng.random(n) > 0.01)
    v = HostColumn.from_numpy(rng.integers(-10**9, 10**9, n), valid=rng.random(n) > 0.05)
    w = HostColumn.from_numpy(rng.standard_normal(n))
    check([key], [(v, INT), (w, [Kind.MIN, Kind.MAX])], NullPolicy.INCLUDE)
    check([key], [(w, [Kind.SUM, Kind.MEAN, Kind.VARIANCE])], NullPolicy.EXCLUDE, row_filters=[v])


# A first table that does not hold the groups: a larger one, a slot per row, up to the rows from which on they are partitioned (one float
# column later than others).
@pytest.mark.parametrize("n,groups,floats,partitioned", [((1 << 18) - 1, 200_000, False, False), (1 << 18, 200_000, False, True),
                                                         ((1 << 19) - 1, 400_000, True, False), (1 << 19, 400_000, True, True)])
def test_the_row_limits(n, groups, floats, partitioned):
    rng = np.random.default_rng(n)
    key = HostColumn.from_numpy(rng.integers(0, groups, n) * 7046029254386353131)
    v = HostColumn.from_numpy(rng.standard_normal(n) if floats else rng.integers(-10**9, 10**9, n))
    check([key], [(v, [Kind.SUM, Kind.MEAN, Kind.VARIANCE] if floats else INT)])
    st = cb.last_call_stats()
    assert st.table_attempts == 2 and (st.table_capacity != int(n / 0.6) + 64) == partitioned


# 2.5M rows, four accumulators: dense ids are partitioned from 25K groups on, others from 69K
@pytest.mark.parametrize("groups,sparse,partitioned", [(12_000, False, False), (50_000, False, True), (40_000, True, False), (150_000, True, True)])
def test_the_sample_decides(groups, sparse, partitioned):
    n = 2_500_000
    rng = np.random.default_rng(groups)
    k = rng.integers(0, groups, n)
    check([HostColumn.from_numpy(k * 7046029254386353131 if sparse else k)], [(HostColumn.from_numpy(rng.integers(-10**9, 10**9, n)), INT)])
    st = cb.last_call_stats()
    assert (st.table_attempts == 1 and st.table_capacity == 1 << 17) != partitioned
