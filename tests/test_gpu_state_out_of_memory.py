"""A state whose table cannot grow keeps its groups.  The allocation that fails is a fake: a preloaded cudaMallocAsync that
refuses requests above a limit."""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

FAKE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static size_t limit = (size_t)-1;
static int refused;
void fake_limit(size_t n) { limit = n; refused = 0; }
int fake_refused(void) { return refused; }
int cudaMallocAsync(void** p, size_t n, void* stream)
{
  static int (*real)(void**, size_t, void*);
  if (!real) real = (int (*)(void**, size_t, void*))dlsym(dlopen("libcudart.so.12", RTLD_NOLOAD | RTLD_LAZY), "cudaMallocAsync");
  if (n > limit) { ++refused; return 2; }
  return real(p, n, stream);
}
"""

USE = r"""
import ctypes, os, sys
import torch
import cudf_b200 as cb
fake = ctypes.CDLL(os.environ["LD_PRELOAD"])
fake.fake_limit.argtypes = [ctypes.c_size_t]
MB = 1 << 20

def batch(lo, n):
    k = (torch.arange(n, device="cuda") + lo) * 1_000_003
    v = torch.arange(n, device="cuda") + lo
    return cb.GroupBy(cb.Table([cb.Column.from_tensor(k)])), [cb.GroupByRequest(cb.Column.from_tensor(v), [cb.aggregation.sum(), cb.aggregation.max()])]

def groups(st):
    k, r = st.finalize()
    n = k.num_rows()
    kk = k.columns()[0].data[:n * 8].view(torch.int64)
    order = torch.argsort(kk)
    assert torch.equal(kk[order], torch.arange(n, device="cuda") * 1_000_003)
    for c in r[0].columns():
        assert torch.equal(c.data[:n * 8].view(torch.int64)[order], torch.arange(n, device="cuda"))
    return n

st = cb.GroupByState(*batch(0, 300_000))
st.update(*batch(0, 300_000))
assert groups(st) == 300_000
# nothing above 4 MB: the table (24 bytes a slot) cannot grow, nor can the batch have one of its own
fake.fake_limit(4 * MB)
for _ in range(2):
    try:
        st.update(*batch(300_000, 600_000))
        raise SystemExit("the update did not fail")
    except MemoryError:
        pass
assert fake.fake_refused() > 0
fake.fake_limit((1 << 64) - 1)
assert st.num_groups() == 300_000 and groups(st) == 300_000
# the state is as good as before
st.update(*batch(300_000, 600_000))
assert groups(st) == 900_000
# memory for a table of the batch's groups, not for one that holds a group per row beside the present one
one = cb.GroupByState(*batch(0, 1000))
one.update(*batch(0, 1000))
fake.fake_limit(24 * MB)

few = cb.GroupBy(cb.Table([cb.Column.from_tensor((torch.arange(2_000_000, device="cuda") % 1000) * 1_000_003)]))
one.update(few, [cb.GroupByRequest(cb.Column.from_tensor(torch.arange(2_000_000, device="cuda") % 1000), [cb.aggregation.sum(), cb.aggregation.max()])])
assert fake.fake_refused() > 0 and one.num_groups() == 1000
fake.fake_limit((1 << 64) - 1)
print("fine")
"""


def test_a_state_that_cannot_grow_keeps_its_groups(tmp_path):
    if not shutil.which("gcc"):
        pytest.skip("needs a C compiler for the fake allocator")
    src, lib = tmp_path / "fake.c", tmp_path / "libfake.so"
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(lib), str(src), "-ldl"], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", USE], cwd=root, env={**os.environ, "LD_PRELOAD": str(lib), "PYTHONPATH": root},
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "fine" in r.stdout, r.stdout + r.stderr
