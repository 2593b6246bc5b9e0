"""The fused pass over a sampled key box with accumulators in their 32-bit forms (b2_box.cuh): value types, nulls, rows that the
sample missed, replicas, tile edges, against the oracle."""
import numpy as np
import pytest

from cudf_b200.types import HostColumn, Kind, NullPolicy
from tests.test_gpu_parity import check

pytestmark = pytest.mark.gpu
TILE = 4096         # rows of one tile of a CTA
AGGS = [Kind.SUM, Kind.MIN, Kind.MAX, Kind.COUNT_VALID, Kind.MEAN]


def _values(rng, dtype, n):
    if np.issubdtype(dtype, np.floating):
        return (rng.standard_normal(n) * 1e3).astype(dtype)
    info = np.iinfo(dtype)
    v = rng.integers(info.min, info.max, n, dtype=dtype, endpoint=True)
    v[::7] = info.max   # (sums carry into the high word, extremes meet the identities of the 32-bit images)
    v[1::11] = info.min
    return v


@pytest.mark.parametrize("dtype", [np.int8, np.uint8, np.int16, np.int32, np.uint32, np.int64, np.uint64, np.float32])
@pytest.mark.parametrize("groups", [1, 70, 3000])
def test_value_types_and_nulls(dtype, groups):
    rng = np.random.default_rng(groups)
    n = 2 * TILE + 777
    k = HostColumn.from_numpy(rng.integers(-groups // 2, groups - groups // 2, n).astype(np.int32))
    x = _values(rng, dtype, n)
    gone = rng.random(n) > 0.4
    gone[k.values() == k.values().min()] = False   # one group without a valid value
    check([k], [(HostColumn.from_numpy(x), AGGS)])
    check([k], [(HostColumn.from_numpy(x), [Kind.MIN, Kind.MAX])])                        # nothing counts the rows
    check([k], [(HostColumn.from_numpy(x, valid=gone), AGGS), (HostColumn.from_numpy(x[::-1].copy()), [Kind.SUM, Kind.MAX])])


@pytest.mark.parametrize("n", [1024, TILE - 1, TILE + 2, 148 * TILE + 1, 149 * TILE - 3])
@pytest.mark.parametrize("width", [np.int8, np.uint16, np.int32, np.int64])
def test_key_widths_tile_edges_and_keys_outside_the_box(width, n):
    rng = np.random.default_rng(n)
    a = rng.integers(0, 50, n).astype(width)
    a[n // 2] = 120                                # (the sample looks at 1024 rows)
    b = HostColumn.from_numpy(rng.integers(0, 5, n).astype(np.int16), valid=rng.random(n) > 0.1)
    v = HostColumn.from_numpy(rng.integers(-10**12, 10**12, n), valid=rng.random(n) > 0.05)
    for policy in (NullPolicy.EXCLUDE, NullPolicy.INCLUDE):
        check([HostColumn.from_numpy(a), b], [(v, AGGS + [Kind.SUM_OF_SQUARES])], policy, row_filters=[v])
        check([HostColumn.from_numpy(a)], [(v, [Kind.COUNT_ALL, Kind.MIN])], policy)
