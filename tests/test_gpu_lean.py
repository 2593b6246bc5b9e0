"""k_aggregate_lean (Σ and n of one float column over a sampled key box): the edges of its tiles, of the window of its
fixed-point sums and of its key box, against the oracle."""
import numpy as np
import pytest

from cudf_b200.types import HostColumn, Kind, NullPolicy
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


def _sums(k, v):
    """Σ by key 0 .. as a host array, in key order."""
    import cudf_b200 as cb
    kt, rt = cb.GroupBy(cb.Table([cb.Column.from_tensor(k)])).aggregate(
        [cb.GroupByRequest(cb.Column.from_tensor(v), [cb.aggregation.sum(), cb.aggregation.count(), cb.aggregation.mean()])])
    order = np.argsort(kt.columns()[0].to_host().values())
    return [c.to_host().values()[order] for c in rt[0].columns()]


@pytest.mark.parametrize("share", [0.005, 0.5])
def test_a_group_of_small_values_beside_a_group_of_large_ones(share):
    """FLOAT64 sums far below the largest one are as exact as any (0.1 beside values near 10^6, 23 binades): a few such rows go
    through the lists, many through the wide window.  A CTA rounds its part of a group's sum once per 1024 addends and at the
    merge: 6M / 1024 + 148 half units of the sum at most, 7e-13, typically their root; every addend rounded gives more than
    10^-12 from 100K addends of one value on."""
    import torch
    n = 12_000_000
    torch.manual_seed(8)
    small = torch.rand(n, device="cuda") < share
    k = torch.where(small, torch.randint(0, 2, (n,), device="cuda"), 2 + torch.randint(0, 20, (n,), device="cuda"))
    tiny, large = torch.tensor([0.1, -0.3], dtype=torch.float64, device="cuda"), 1e6 + torch.rand(n, dtype=torch.float64, device="cuda")
    v = torch.where(small, tiny[k.clamp(max=1)], large)
    s, c, m = _sums(k, v)
    for g, x in ((0, 0.1), (1, -0.3)):
        assert c[g] == int((small & (k == g)).sum())
        assert abs(s[g] - x * c[g]) <= 3e-14 * abs(x * c[g])
        assert abs(m[g] - x) <= 3e-14 * abs(x)


@pytest.mark.parametrize("big", [1e9, 1e300, 1e-300])
def test_unsampled_magnitudes(big):
    """A group of values that no sampled row has, far above or below all others."""
    import torch
    n = 2_000_000
    rng = np.random.default_rng(9)
    i = np.arange(1024)
    free = np.ones(n, dtype=bool)
    free[i * (n // 1024) + (i * 7919) % (n // 1024)] = False
    pick = free & (rng.random(n) < 0.02)
    k = np.where(pick, 7, rng.integers(0, 7, n))
    x = rng.random(n) + 1
    x[pick] = big * (1 + rng.random(int(pick.sum())))
    s, c, _ = _sums(torch.from_numpy(k).cuda(), torch.from_numpy(x).cuda())
    for g in range(8):
        import math
        exact = math.fsum(x[k == g])
        assert c[g] == int((k == g).sum()) and abs(s[g] - exact) <= 2e-14 * abs(exact)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("share", [1e-5, 0.3])
def test_infinities_and_nans(dtype, share):
    rng = np.random.default_rng(10)
    n = 500_003
    k = rng.integers(0, 6, n).astype(np.int64)
    x = rng.standard_normal(n).astype(dtype)
    odd = rng.random(n) < share
    odd[rng.integers(0, n, 40)] = True
    for g, values in enumerate(([np.inf], [-np.inf], [np.inf, -np.inf], [np.nan], [np.nan, np.inf])):
        at = np.flatnonzero(odd & (k == g))
        x[at] = np.resize(np.array(values, dtype=dtype), at.size)
    for valid in (None, rng.random(n) > 0.1):
        v = HostColumn.from_numpy(x, valid=valid)
        check([HostColumn.from_numpy(k)], [(v, AGGS)])
        check([HostColumn.from_numpy(k)], [(v, [Kind.MEAN])], row_filters=[v] if valid is not None else [])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("variant", [0, 4])
@pytest.mark.parametrize("groups", [3, 1000, 9000, 12_500])
def test_values_over_many_binades(dtype, variant, groups):
    """Log-normal values of sigma 3: the wide window, with the tile ring or register tiles as the box leaves room, or, beyond
    that, the generic kernel; one and two key columns, key masks, row counts around the tiles."""
    rng = np.random.default_rng(groups)
    for n in (200 * TILE + 3, 40 * TILE + 4095):
        x = (rng.lognormal(0, 3, n) * rng.choice([-1, 1], n)).astype(dtype)
        v = HostColumn.from_numpy(x, valid=rng.random(n) > 0.05)
        k = rng.integers(0, groups, n)
        check([HostColumn.from_numpy(k.astype(np.int64))], [(v, AGGS)], table_variant=variant)
        check([HostColumn.from_numpy((k // 50).astype(np.int32)), HostColumn.from_numpy((k % 50).astype(np.int32), valid=rng.random(n) > 0.05)],
              [(v, [Kind.MEAN])], NullPolicy.INCLUDE, row_filters=[v], table_variant=variant)
