"""Packed keys whose table of the first attempt does not hold the groups, around the rows from which on they are partitioned, and
inputs that the sample sends there at once: against the oracle."""
import numpy as np
import pytest

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
