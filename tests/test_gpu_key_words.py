"""The partitioned path over keys told by 32-bit words (b2_partition.cuh): key types, strides, nulls and outliers of the sampled
box, records of 4- and 8-byte values with and without validity, one and two levels of digits, against the oracle."""
import numpy as np
import pytest

from cudf_b200.types import HostColumn, Kind, NullPolicy
from tests.test_gpu_parity import check

pytestmark = pytest.mark.gpu
INT = [Kind.SUM, Kind.MIN, Kind.MAX, Kind.COUNT_VALID]
TILE = 4096
BOTH = pytest.mark.parametrize("table_bytes", [0, 16384])   # 16 KB tables: two levels


def _column(x, valid=None):
    return HostColumn.from_numpy(x, valid=valid)


@BOTH
@pytest.mark.parametrize("dtype", [np.int16, np.uint16, np.int32, np.uint32, np.int64, np.uint64])
@pytest.mark.parametrize("first", [0, -20_000, 40_000])
def test_key_types_and_where_the_box_lies(dtype, first, table_bytes):
    info = np.iinfo(dtype)
    if first < info.min or first + 20_000 > info.max:
        first = info.max - 20_000 if first > 0 else info.min
    rng = np.random.default_rng(3)
    n = 20 * TILE + 5
    k = (rng.integers(0, 20_001, n) + int(first)).astype(dtype)
    v = rng.integers(-10**9, 10**9, n)
    check([_column(k)], [(_column(v), INT)], table_variant=6, shared_table_bytes=table_bytes)
    check([_column(k, rng.random(n) > 0.1)], [(_column(v, rng.random(n) > 0.2), INT)], NullPolicy.INCLUDE if k.itemsize < 8 else NullPolicy.EXCLUDE,
          table_variant=6, shared_table_bytes=table_bytes)


@BOTH
@pytest.mark.parametrize("stride,groups", [(1, 300_000), (2, 150_000), (64, 9_000), (1 << 18, 3), (999, 700)])
def test_strides_of_ids(stride, groups, table_bytes):
    rng = np.random.default_rng(stride)
    n = 700_001
    k = rng.integers(0, groups, n) * stride
    check([_column(k)], [(_column(rng.integers(0, 100, n).astype(np.int32)), INT)], table_variant=6, shared_table_bytes=table_bytes)


@pytest.mark.parametrize("outlier", [-1, -2**62, 30_000_000, 2**31, 2**40, 2**63 - 1])
@pytest.mark.parametrize("low", [0, 1_000_000])
def test_a_key_that_the_sample_did_not_show(outlier, low):
    """Below the first position, beyond 32 bits, or so far above that the box grows too large: hashed keys instead."""
    rng = np.random.default_rng(5)
    n = 300_000
    k = rng.integers(low, low + 50_000, n)
    k[n // 2 + 1] = outlier
    check([_column(k)], [(_column(rng.integers(-5, 5, n)), INT)], table_variant=6)
    check([_column(k)], [(_column(rng.standard_normal(n)), [Kind.SUM, Kind.MEAN, Kind.VARIANCE])], table_variant=6)


@BOTH
@pytest.mark.parametrize("policy", [NullPolicy.EXCLUDE, NullPolicy.INCLUDE])
def test_two_key_columns(policy, table_bytes):
    rng = np.random.default_rng(6)
    n = 30 * TILE - 1
    a = _column(rng.integers(-300, 300, n).astype(np.int32), rng.random(n) > 0.05)
    b = _column(rng.integers(0, 90, n).astype(np.int16), rng.random(n) > 0.05)
    v = _column(rng.standard_normal(n).astype(np.float32), rng.random(n) > 0.3)
    check([a, b], [(v, INT + [Kind.MEAN]), (_column(rng.integers(0, 2**40, n)), INT)], policy, table_variant=6, shared_table_bytes=table_bytes)
    check([b, a], [(v, [Kind.MEAN])], policy, row_filters=[v], table_variant=6, shared_table_bytes=table_bytes)


@BOTH
@pytest.mark.parametrize("top", [100, 2**31 - 1, 2**31, 2**32 - 1, 2**32, 2**63 - 1])
@pytest.mark.parametrize("least", [0, -1, -2**31, -2**31 - 1])
def test_values_at_the_edges_of_32_bits(top, least, table_bytes):
    rng = np.random.default_rng(7)
    n = 300_003
    v = rng.integers(0, 100, n)
    v[5::1000] = top
    v[6::1000] = least
    k = rng.integers(0, 70_000, n)
    check([_column(k)], [(_column(v), INT)], table_variant=6, shared_table_bytes=table_bytes, expected_groups=400_000)
    check([_column(k)], [(_column(v, rng.random(n) > 0.3), [Kind.MIN, Kind.MAX])], table_variant=6, shared_table_bytes=table_bytes,
          expected_groups=400_000)


@BOTH
@pytest.mark.parametrize("n", [1024, TILE - 3, TILE, TILE + 1, 149 * TILE + 2])
def test_ragged_sizes_and_groups_without_values(n, table_bytes):
    rng = np.random.default_rng(n)
    k = rng.integers(10, 10 + n // 3, n).astype(np.int32)
    gone = rng.random(n) > 0.3
    gone[k < 20] = False
    for v in (rng.standard_normal(n), rng.standard_normal(n).astype(np.float32)):
        check([_column(k)], [(_column(v, gone), [Kind.SUM, Kind.MEAN, Kind.VARIANCE])], table_variant=6, shared_table_bytes=table_bytes)
        check([_column(k)], [(_column(v), [Kind.SUM])], table_variant=6, shared_table_bytes=table_bytes)
        check([_column(k)], [(_column(v, gone), [Kind.MIN, Kind.MAX]), (_column(k), [Kind.COUNT_ALL])], table_variant=6, shared_table_bytes=table_bytes)
    fifteen = [(_column(rng.integers(0, 9, n).astype(np.int8), rng.random(n) > 0.5), [Kind.MAX]) for _ in range(15)]
    check([_column(k)], fifteen, table_variant=6)   # (validity bits in an array: the word has no room for 15)


def test_many_rows_few_groups_straight_into_the_columns():
    rng = np.random.default_rng(8)
    n = 5_000_003
    k = rng.integers(0, 300_000, n).astype(np.int64)
    k[k > 100_000] = 7 * (k[k > 100_000] // 7)          # (a good part of the box stays empty)
    v = _column(rng.integers(-1000, 1000, n), rng.random(n) > 0.05)
    check([_column(k)], [(v, INT + [Kind.VARIANCE])])
