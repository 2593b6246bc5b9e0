"""Wide keys whose dictionary or ids do not fit memory are grouped as row keys.  The allocation that fails is a fake: a preloaded
cudaMallocAsync that refuses requests above a limit."""
import os
import shutil
import subprocess
import sys

import pytest

from tests.test_gpu_state_out_of_memory import FAKE

pytestmark = pytest.mark.gpu

USE = r"""
import ctypes, os
import torch
import cudf_b200 as cb
fake = ctypes.CDLL(os.environ["LD_PRELOAD"])
fake.fake_limit.argtypes = [ctypes.c_size_t]
MB = 1 << 20
n, groups = 4_400_000, 100_000          # enough rows and few enough groups for ids (17.6 MB), whose dictionary has 48 MB
g = torch.randint(0, groups, (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
g[:groups] = torch.arange(groups, device="cuda")
v = torch.arange(n, device="cuda") % 1000
keys = cb.Table([cb.Column.from_tensor(g * 1_000_003), cb.Column.from_tensor((g % 7).to(torch.int32))])
reqs = [cb.GroupByRequest(cb.Column.from_tensor(v), [cb.aggregation.sum(), cb.aggregation.max(), cb.aggregation.count()])]
want = torch.zeros(groups, dtype=torch.int64, device="cuda").index_add_(0, g, v)
for limit in (1 << 40, 32 * MB, 16 * MB):
    fake.fake_limit(limit)
    k, (r,) = cb.GroupBy(keys).aggregate(reqs)
    refused = fake.fake_refused()
    assert (refused > 0) == (limit < 1 << 40), (limit, refused)
    assert k.num_rows() == groups
    at = k.columns()[0].data[:groups * 8].view(torch.int64) // 1_000_003
    assert torch.equal(k.columns()[1].data[:groups * 4].view(torch.int32).to(torch.int64), at % 7)
    assert torch.equal(torch.zeros_like(want).scatter_(0, at, r.columns()[0].data[:groups * 8].view(torch.int64)), want)
print("fine")
"""


def test_wide_keys_without_memory_for_ids(tmp_path):
    if not shutil.which("gcc"):
        pytest.skip("needs a C compiler for the fake allocator")
    src, lib = tmp_path / "fake.c", tmp_path / "libfake.so"
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(lib), str(src), "-ldl"], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", USE], cwd=root, env={**os.environ, "LD_PRELOAD": str(lib), "PYTHONPATH": root},
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "fine" in r.stdout, r.stdout + r.stderr
