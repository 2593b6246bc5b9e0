"""Key columns that do not pack into 64 bits, told by dictionary ids (k_dict_encode over fixed-width columns): against the
oracle.  table_variant 8 takes that way whatever the number of rows."""
import numpy as np
import pytest

from cudf_b200.types import HostColumn, Kind, NullPolicy
from tests.test_gpu_parity import check

pytestmark = pytest.mark.gpu
AGGS = [Kind.SUM, Kind.MIN, Kind.MAX, Kind.MEAN, Kind.COUNT_VALID]
BOTH = pytest.mark.parametrize("policy", [NullPolicy.EXCLUDE, NullPolicy.INCLUDE])


def _col(x, valid=None, offset=0):
    return HostColumn.from_numpy(x, valid=valid, offset=offset)


@BOTH
@pytest.mark.parametrize("n", [1, 31, 1023, 1025, 60_001])
def test_composites_with_nulls_and_filters(n, policy):
    rng = np.random.default_rng(n)
    a = _col(rng.integers(-2**62, 2**62, 50)[rng.integers(0, 50, n)], rng.random(n) > 0.1, offset=3)
    b = _col(rng.integers(0, 9, n).astype(np.int32), rng.random(n) > 0.1)
    c = _col(rng.integers(0, 3, n).astype(np.int8))
    v = _col(rng.standard_normal(n), rng.random(n) > 0.2)
    check([a, b, c], [(v, AGGS)], policy, table_variant=8)
    check([c, b, a], [(v, AGGS + [Kind.ARGMIN])], policy, row_filters=[v], table_variant=8)


@BOTH
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_float_keys(dtype, policy):
    rng = np.random.default_rng(2)
    n = 20_003
    pool = np.concatenate([rng.standard_normal(100), [0.0, np.nan, np.inf, -np.inf]]).astype(dtype)
    k = _col(pool[rng.integers(0, pool.size, n)], rng.random(n) > 0.05)
    check([k], [(_col(rng.integers(0, 100, n)), AGGS)], policy, table_variant=8)
    check([k, _col(rng.integers(0, 4, n).astype(np.int16))], [(_col(rng.integers(0, 100, n)), AGGS)], policy, table_variant=8)


def test_widest_and_too_wide():
    rng = np.random.default_rng(3)
    n = 5_000
    cols = [_col(rng.integers(0, 3, n)) for _ in range(5)]
    v = _col(rng.integers(0, 100, n).astype(np.int32))
    for m in (3, 4, 5):     # 24 bytes; 32 bytes and 40 bytes go the way of row keys
        check(cols[:m], [(v, AGGS)], table_variant=8)


@pytest.mark.parametrize("groups", [3, 40_000, 900_000])
def test_many_rows(groups):
    """Few groups (every CTA inserts the same keys at once), some, and so many that the first dictionary is too small."""
    rng = np.random.default_rng(groups)
    n = 1_200_007
    g = rng.integers(0, groups, n)
    a, b = _col(g * 1_000_003), _col((g % 7).astype(np.int32), rng.random(n) > 0.01)
    check([a, b], [(_col(rng.integers(-50, 50, n)), AGGS)], NullPolicy.INCLUDE, table_variant=8)
    check([_col(g * 0.5)], [(_col(rng.integers(-50, 50, n)), AGGS)], table_variant=8)


@pytest.mark.parametrize("groups", [250_000, 900_000])
@pytest.mark.parametrize("n", [1_200_007, 300 * 1024 + 1])
def test_a_dictionary_that_overflows_with_rows_left_out(n, groups):
    """Null keys under EXCLUDE (a ballot per tile notes the rows that take part) while CTAs stop because the first table is full."""
    rng = np.random.default_rng(n + groups)
    g = rng.integers(0, groups, n)
    a, b = _col(g * 1_000_003, rng.random(n) > 0.03), _col((g % 7).astype(np.int32), rng.random(n) > 0.02)
    v = _col(rng.integers(-50, 50, n))
    check([a, b], [(v, AGGS)], NullPolicy.EXCLUDE, table_variant=8)
    check([_col(g * 0.5, rng.random(n) > 0.03)], [(v, AGGS)], NullPolicy.EXCLUDE, row_filters=[b], table_variant=8)


@pytest.mark.parametrize("groups", [10, 500, 60_000, 2_000_000])
def test_the_sample_decides(groups):
    """Enough rows for the automatic choice: the cache of the row-key pass, ids over a key box, ids through partitions, row keys."""
    rng = np.random.default_rng(groups)
    n = (1 << 22) + 11
    g = rng.integers(0, groups, n)
    check([_col(g * 1_000_003), _col((g % 7).astype(np.int32))], [(_col(rng.integers(-50, 50, n)), [Kind.SUM, Kind.MIN, Kind.COUNT_VALID])])


@pytest.mark.parametrize("aggs", [[Kind.COUNT_VALID], [Kind.MEAN, Kind.MIN]])
@pytest.mark.parametrize("groups", [300, 900, 50_000, 120_000])
def test_the_sample_decides_about_one_key_column(groups, aggs):
    """Both sides of the two lines for a single column: groups that a cache holds, and rows for every group of a lone accumulator."""
    rng = np.random.default_rng(groups)
    n = (1 << 22) + 11
    check([_col(rng.integers(0, groups, n) * 0.5, rng.random(n) > 0.01)], [(_col(rng.integers(-50, 50, n).astype(np.int32)), aggs)])
