"""k_aggregate_lean (Σ and n of one float column over a sampled key box): the edges of its tiles, of the window of its
fixed-point sums and of its key box, against the oracle."""
import numpy as np
import pytest

from cudf_b200.types import HostColumn, Kind
from tests.test_gpu_parity import check

pytestmark = pytest.mark.gpu
AGGS = [Kind.SUM, Kind.COUNT_VALID, Kind.MEAN]
TILE = 992 * 4      # rows of one tile of the ring


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1024, 4 * TILE - 1, 4 * TILE, 4 * TILE + 3, 149 * TILE + 5, 300 * TILE + TILE - 4])
def test_rows_around_tile_edges(dtype, n):
    rng = np.random.default_rng(n)
    k = HostColumn.from_numpy(rng.integers(-20, 20, n).astype(np.int32))
    v = HostColumn.from_numpy((rng.standard_normal(n) * 7).astype(dtype), valid=rng.random(n) > 0.1)
    check([k], [(v, AGGS)])
    check([k], [(v, [Kind.MEAN])], row_filters=[v])
    check([k], [(HostColumn.from_numpy((rng.random(n) * 7).astype(dtype)), AGGS)], table_variant=4)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_values_outside_the_window(dtype):
    """Magnitudes over 60 binades, signed zeros, denormals; few groups, so that slots fill up and are emptied."""
    rng = np.random.default_rng(11)
    n = 700_001
    k = rng.integers(0, 6, n).astype(np.int64)
    x = (rng.standard_normal(n) * np.exp2(rng.integers(-40, 20, n))).astype(dtype)
    x[k == 1] = 0.0
    x[k == 2] = np.abs(x[k == 2])
    x[(k == 3) & (rng.random(n) < 0.2)] = -0.0
    x[k == 4] = np.finfo(dtype).smallest_subnormal
    v = HostColumn.from_numpy(x, valid=rng.random(n) > 0.02)
    check([HostColumn.from_numpy(k)], [(v, AGGS)])


@pytest.mark.parametrize("share", [0.001, 0.05, 0.4])
def test_keys_outside_the_box(share):
    """Rows whose key the sample did not span: a few (listed and worked off behind the row loop), and so many that the
    lists overflow or no box fits and another kernel takes the input."""
    rng = np.random.default_rng(12)
    n = 600_000
    far = rng.random(n) < share
    k = np.where(far, rng.integers(10**6, 10**6 + 3000, n), rng.integers(0, 200, n)).astype(np.int64)
    v = HostColumn.from_numpy(rng.random(n).astype(np.float32) * 100, valid=rng.random(n) > 0.05)
    check([HostColumn.from_numpy(k)], [(v, AGGS)])
    k[far] = 10**12
    check([HostColumn.from_numpy(k)], [(v, AGGS)])
    # far keys in a part of the input that is not sampled at all: one row in 585 is
    k = rng.integers(0, 200, n).astype(np.int64)
    stride = n // 1024
    i = np.arange(1024)
    sampled = i * stride + (i * 7919) % stride
    free = np.ones(n, dtype=bool)
    free[sampled] = False
    pick = free & (rng.random(n) < share)
    k[pick] = rng.integers(10**9, 10**9 + 50, int(pick.sum()))
    check([HostColumn.from_numpy(k)], [(v, AGGS)])


@pytest.mark.parametrize("variant", [0, 4])   # 0: tile ring, 4: register tiles
@pytest.mark.parametrize("lo,rare", [(0, 2**32 - 1), (2**32 - 1000, 0), (-2**31, 2**31 - 1), (2**31 - 1000, -2**31)])
def test_key_boxes_at_the_ends_of_a_type(lo, rare, variant):
    """1000 ids at one end of a 32-bit type and a few rows at the other, among the full tiles and behind them: modulo 2^32
    the two are neighbours, and a box padded across the end would give the rare key two groups."""
    n = 30 * TILE + (4095 if variant else 3)
    rng = np.random.default_rng(3)
    dt = np.int32 if lo < 0 or rare < 0 else np.uint32
    stride = n // 1024
    i = np.arange(1024)
    free = np.ones(n, dtype=bool)
    free[i * stride + (i * 7919) % stride] = False   # (the rows the key-box sampler looks at)
    k = lo + rng.integers(0, 1000, n)
    for part in (np.flatnonzero(free[:n // 2]), n - 5 + np.flatnonzero(free[n - 5:])):
        k[part[-3:]] = rare
    v = HostColumn.from_numpy(rng.random(n), valid=rng.random(n) > 0.1)
    check([HostColumn.from_numpy(k.astype(dt))], [(v, AGGS)], table_variant=variant)
    check([HostColumn.from_numpy(k.astype(dt))], [(HostColumn.from_numpy(rng.random(n).astype(np.float32)), AGGS)], table_variant=variant)


@pytest.mark.parametrize("n", [1024, 4095, 4096, 4097])
def test_small_float64_sums_are_rounded_once(n):
    """Σ of one FLOAT64 column on both sides of the line between k_small and the lean kernel: within one unit of the last place
    of the exact sum (exact fixed point, or two doubles that together hold 106 bits)."""
    import math
    import cudf_b200 as cb
    import torch
    rng = np.random.default_rng(n)
    for x in (np.full(n, 0.1), rng.lognormal(0, 2, n), rng.standard_normal(n) + 100):
        for keys in (np.zeros(n), np.arange(n) % 7):
            k = cb.Column.from_tensor(torch.from_numpy(keys.astype(np.int64)).cuda())
            v = cb.Column.from_tensor(torch.from_numpy(x).cuda())
            kt, rt = cb.GroupBy(cb.Table([k])).aggregate([cb.GroupByRequest(v, [cb.aggregation.sum(), cb.aggregation.mean()])])
            got_k, got = kt.columns()[0].to_host().values(), rt[0].columns()[0].to_host().values()
            for g, s in zip(got_k, got):
                exact = math.fsum(x[keys == g])
                assert abs(s - exact) <= 2.0 ** -52 * abs(exact)
