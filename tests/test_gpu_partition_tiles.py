"""``hash_partition`` through tiles sorted in shared memory (9 to 512 partitions): the edges of that range, STRING columns beside
fixed-width ones and alone (a permutation), several tiles per CTA, against the oracle's assignment."""
import numpy as np
import pytest
import torch

from cudf_b200.types import HostColumn, TypeId
from tests.test_gpu_partition import _mixed_table, _table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nparts", [23, 24, 200, 511, 512, 513])
@pytest.mark.parametrize("n", [1, 4095, 8193, 20_000])
def test_strings_and_fixed_columns(n, nparts):
    from cudf_b200.partition import hash_partition
    from oracle import partition_oracle as PO
    mixed = _mixed_table(n + nparts, n)
    number = HostColumn.from_strings([str(i) for i in range(n)])
    for cols, hashed in ((mixed + [number], [0, 3]), ([mixed[1], mixed[3], number], [1])):   # (strings only: nothing but the permutation)
        out, offsets = hash_partition(_table(cols), hashed, nparts)
        got = [c.to_host() for c in out.columns()]
        rows = np.array([int(x) for x in got[-1].to_pylist()], dtype=np.int64)
        part = PO.partition_of_rows([cols[i] for i in hashed], nparts)
        assert np.array_equal(np.sort(rows), np.arange(n)) and np.array_equal(np.diff(offsets), np.bincount(part, minlength=nparts))
        assert np.array_equal(part[rows], np.repeat(np.arange(nparts), np.diff(offsets)))
        for g, c in zip(got, cols):
            src = c.to_pylist()
            assert [repr(x) for x in g.to_pylist()] == [repr(src[i]) for i in rows] and g.null_count == c.null_count


@pytest.mark.parametrize("nparts", [8, 9, 16, 23, 512])
def test_several_tiles_per_cta(nparts):
    """From 2^22 rows on the tiles begin at 9 partitions.  A string holds its row's number, and so does a column."""
    import cudf_b200 as cb
    from cudf_b200.partition import hash_partition
    from oracle import partition_oracle as PO
    n = (1 << 22) + 4097
    rng = np.random.default_rng(nparts)
    key = HostColumn.from_numpy(rng.integers(0, 10**6, n), valid=rng.random(n) > 0.02)
    narrow = HostColumn.from_numpy(rng.integers(0, 30_000, n).astype(np.int16), valid=rng.random(n) > 0.5)
    number = torch.arange(n, dtype=torch.int32, device="cuda")
    text = cb.Column(TypeId.STRING, n, number.view(torch.uint8).clone(), None, 0, 0,
                     (torch.arange(n + 1, dtype=torch.int32, device="cuda") * 4).view(torch.uint8), TypeId.INT32)
    fixed = [cb.Column.from_host(key), cb.Column.from_host(narrow), cb.Column.from_tensor(number)]
    part = PO.partition_of_rows([key], nparts)
    for columns in (fixed, fixed + [text], [fixed[0], text]):
        out, offsets = hash_partition(cb.Table(columns), [0], nparts)
        got = out.columns()
        if columns[-1] is text:
            assert torch.equal(got[-1].offsets.view(torch.int32)[:n + 1], torch.arange(n + 1, dtype=torch.int32, device="cuda") * 4)
            rows = got[-1].data[:4 * n].view(torch.int32).cpu().numpy()
        else:
            rows = got[2].data[:4 * n].view(torch.int32).cpu().numpy()
        assert np.array_equal(np.sort(rows), np.arange(n))
        assert np.array_equal(np.diff(offsets), np.bincount(part, minlength=nparts))
        assert np.array_equal(part[rows], np.repeat(np.arange(nparts), np.diff(offsets)))
        for c, src in zip(got[:2], (key, narrow) if len(columns) > 2 else (key,)):
            h = c.to_host()
            assert np.array_equal(h.valid(), src.valid()[rows]) and h.null_count == src.null_count
            assert np.array_equal(h.values()[h.valid()], src.values()[rows][h.valid()])
        if len(columns) == 4:
            assert np.array_equal(got[2].data[:4 * n].view(torch.int32).cpu().numpy(), rows)
