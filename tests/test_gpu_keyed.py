"""Keys that do not pack, aggregated in the pass that tells them apart (k_keyed; table_variant 9 takes it whatever the number of
rows): against the oracle."""
import numpy as np
import pytest

from cudf_b200.types import HostColumn, Kind, NullPolicy, TypeId
from tests.test_gpu_parity import check

pytestmark = pytest.mark.gpu
AGGS = [Kind.SUM, Kind.MIN, Kind.MAX, Kind.MEAN, Kind.COUNT_VALID, Kind.VARIANCE]
BOTH = pytest.mark.parametrize("policy", [NullPolicy.EXCLUDE, NullPolicy.INCLUDE])


def _col(x, valid=None, offset=0):
    return HostColumn.from_numpy(x, valid=valid, offset=offset)


def _strings(rng, n, pool, nulls=0.0, large=False):
    words = ["", "a", "ab", "año", "q" * 31, "q" * 32, "q" * 33, "q" * 32 + "x", "z" * 300] + ["key%d" % i * (1 + i % 5) for i in range(pool)]
    return HostColumn.from_strings([None if rng.random() < nulls else words[i] for i in rng.integers(0, len(words), n)], large_offsets=large)


# edges of a warp, a CTA and a grid, more groups than a CTA's accumulators
@BOTH
@pytest.mark.parametrize("n,pool", [(1, 1), (33, 5), (513, 40), (70_001, 3), (70_001, 30_000), (700_003, 200)])
def test_strings(n, pool, policy):
    rng = np.random.default_rng(n + pool)
    s = _strings(rng, n, pool, 0.05, large=n % 2 == 0)
    v = _col(rng.integers(-1000, 1000, n).astype(np.int32), rng.random(n) > 0.1)
    w = _col(rng.standard_normal(n).astype(np.float32))
    check([s], [(v, AGGS), (w, [Kind.MIN, Kind.MAX])], policy, table_variant=9)
    k = _col(rng.integers(0, 3, n).astype(np.int16), rng.random(n) > 0.1)
    check([k, s], [(w, AGGS)], policy, row_filters=[v], table_variant=9)


@BOTH
@pytest.mark.parametrize("n,groups", [(1, 1), (513, 40), (70_001, 4), (300_007, 60_000)])
def test_fixed_width(n, groups, policy):
    rng = np.random.default_rng(n)
    g = rng.integers(0, groups, n)
    a, b = _col(g * 1_000_000_007, rng.random(n) > 0.02, offset=3), _col((g % 7).astype(np.int32), rng.random(n) > 0.02)
    v, w = _col(rng.standard_normal(n), rng.random(n) > 0.2), _col(rng.integers(-2**62, 2**62, n))
    check([a, b], [(v, AGGS), (w, [Kind.SUM, Kind.MIN, Kind.MAX, Kind.COUNT_ALL])], policy, table_variant=9)
    pool = np.concatenate([rng.standard_normal(groups), [0.0, -0.0, np.nan, np.inf, -np.inf]])
    check([_col(pool[rng.integers(0, pool.size, n)], rng.random(n) > 0.05)], [(v, AGGS)], policy, row_filters=[v], table_variant=9)


@pytest.mark.parametrize("dtype", [np.int8, np.uint16, np.int32, np.uint32, np.float32, np.int64])
def test_extremes_of_the_type(dtype):
    """A group whose only value is what an empty accumulator holds."""
    n = 5_000
    rng = np.random.default_rng(1)
    info = np.finfo(dtype) if dtype == np.float32 else np.iinfo(dtype)
    g = rng.integers(0, 6, n)
    x = np.array([info.max, info.min, 0, 1, info.max, info.min], dtype)[g]
    for valid in (None, rng.random(n) > 0.5):
        check([_col(g * 0.5)], [(_col(x, valid), [Kind.MIN, Kind.MAX])], table_variant=9)


def test_what_it_does_not_serve():
    """Two STRING columns, keys beyond an entry, row indices as results, more distinct keys than its dictionary holds: the ways that
    served them before."""
    rng = np.random.default_rng(5)
    n = 20_000
    s, t = _strings(rng, n, 10), _strings(rng, n, 10)
    v = _col(rng.integers(0, 100, n).astype(np.int32))
    check([s, t], [(v, AGGS)], table_variant=9)
    check([_col(rng.integers(0, 3, n)) for _ in range(5)], [(v, AGGS)], table_variant=9)
    check([s, _col(rng.integers(0, 3, n)), _col(rng.integers(0, 3, n).astype(np.int8))], [(v, AGGS)], table_variant=9)
    check([s], [(v, [Kind.ARGMIN])], table_variant=9)
    m = 3_500_000
    check([_col(np.arange(m) * 0.5)], [(_col(np.ones(m, np.int32)), [Kind.SUM])], table_variant=9)


def test_nothing_left():
    one = _col(np.ones(1000, np.int32))
    nothing = HostColumn.from_strings([None] * 1000)
    assert check([nothing], [(one, [Kind.SUM])], NullPolicy.EXCLUDE, table_variant=9)[0][0].size == 0
    assert check([nothing], [(one, [Kind.SUM])], NullPolicy.INCLUDE, table_variant=9)[0][0].size == 1
