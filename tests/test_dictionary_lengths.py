"""What the dictionary of STRING keys makes of a string's length, on the host: strings of 2 and 4 GiB and more are not taken for
short ones or for ones of negative length.  (A call with such a string would hash and compare gigabytes in one thread.)"""
import os
import subprocess

import pytest

from cudf_b200.build import HERE, find_nvcc

PROGRAM = r"""
#include "b2_device.cuh"
#include <cstdio>
using namespace b2;
int main()
{
  const u64 h = 0xFEDCBA9876543210ull;
  const i64 lengths[] = {0, 5, 31, 32, 33, 253, 254, 255, (1ll << 31) - 1, 1ll << 31, (1ll << 32) - 1, 1ll << 32, (1ll << 32) + 5, 1ll << 40};
  for (i64 n : lengths) {
    const int bytes = dict_length(n);
    const u64 head = dict_head(h, bytes);
    const bool ok = bytes == (n < 0x7FFFFFFF ? n : 0x7FFFFFFF) && (bytes > DICT_INLINE) == (n > DICT_INLINE) && dict_kept(bytes) == (n < 32 ? n : 32) &&
                    (head >> 34) == (h >> 34) && ((head >> 26) & 0xFF) == (u64)(n < 254 ? n : 254) && (head & DICT_ID_MASK) == 0;
    if (!ok) { std::printf("length %lld\n", (long long)n); return 1; }
  }
  return 0;
}
"""


def test_lengths_of_strings(tmp_path):
    try:
        nvcc = find_nvcc()
    except RuntimeError:
        pytest.skip("needs nvcc")
    src, exe = tmp_path / "lengths.cu", tmp_path / "lengths"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", os.path.join(HERE, "csrc"), "-o", str(exe), str(src)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
