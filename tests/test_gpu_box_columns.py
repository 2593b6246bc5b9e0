"""The pass over a key box, column by column (sums, counts, minima and maxima): value types and forms, extremes that an empty cell
holds, rows outside the box or without a key, whose cells are looked at all the same."""
import numpy as np
import pytest

from cudf_b200.types import HostColumn, Kind, NullPolicy
from tests.test_gpu_parity import check

pytestmark = pytest.mark.gpu
AGGS = [Kind.SUM, Kind.MIN, Kind.MAX, Kind.COUNT_VALID]
TYPES = [np.int8, np.uint16, np.int32, np.uint32, np.int64, np.uint64, np.float32, np.float64]


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("n,groups", [(4097, 3), (70_001, 2000)])
def test_types(n, groups, dtype):
    rng = np.random.default_rng(n)
    info = np.finfo(dtype) if np.issubdtype(dtype, np.floating) else np.iinfo(dtype)
    x = (rng.standard_normal(n) * 50).astype(dtype) if np.issubdtype(dtype, np.floating) else rng.integers(info.min, info.max, n, dtype, endpoint=True)
    g = rng.integers(0, groups, n)
    x[g == 0], x[g == 1] = info.max, info.min
    sums = AGGS if dtype not in (np.float32, np.float64) else [Kind.MIN, Kind.MAX, Kind.COUNT_VALID]
    far = g.astype(np.int64)
    far[rng.choice(n, 5, replace=False)] = 2**40   # outside the box, or its type's whole range
    k = HostColumn.from_numpy(far, valid=rng.random(n) > 0.02)
    for valid in (None, rng.random(n) > 0.3):
        v = HostColumn.from_numpy(x, valid=valid)
        w = HostColumn.from_numpy(rng.integers(-9, 9, n).astype(np.int32))
        check([k], [(v, sums)], NullPolicy.EXCLUDE)
        check([k], [(v, sums), (w, AGGS + [Kind.COUNT_ALL])], NullPolicy.INCLUDE, row_filters=[v] if valid is not None else [])
