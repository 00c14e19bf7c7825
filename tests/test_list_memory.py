"""Device memory of the calls that keep buffers: a long list takes what its
primes need, not what a window of its width could hold, and a call that runs out
of memory goes again without the buffers that were kept."""
import os
import shutil
import subprocess
import sys

import pytest

from conftest import ROOT

# [9 * 10^13, + 2 * 10^8): 6.2 million primes (50 MB) and 6.7 MB of bitmap, each
# with an eighth more; room for the 2.1 * 10^7 primes that fit a window of that
# width at most would be 167 MB.
GROWTH = r"""
import ctypes
import torch
from voss_gb300 import _capi

def listed(width):
    arr, n = ctypes.POINTER(ctypes.c_uint64)(), ctypes.c_uint64()
    a = 9 * 10**13
    assert _capi._lib.voss_primes_in_range_with_limit(a, a + width, 10**9, ctypes.byref(arr), ctypes.byref(n)) == 0
    _capi._lib.voss_free(arr)
    return n.value

listed(12 * 10**8)          # over 256 MB: nothing of it stays but the prime table and the driver's own
before = torch.cuda.mem_get_info()[0]
print(listed(2 * 10**8), (before - torch.cuda.mem_get_info()[0]) >> 20)
"""


@pytest.mark.gpu
def test_a_long_list_takes_what_it_holds(vg, oracle_lib):
    out = subprocess.run([sys.executable, "-c", GROWTH], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    n, mb = map(int, out.stdout.split())
    assert n == len(oracle_lib.primes_in_range(9 * 10**13, 9 * 10**13 + 2 * 10**8))
    assert mb <= 80, mb


@pytest.mark.gpu
@pytest.mark.parametrize("a", [0, 10**11])
def test_lists_on_both_sides_of_the_room(vg, oracle_lib, a):
    # 2 w / ln w primes of 8 bytes pass 144 MB at a width of 1.794 * 10^8
    for width in (179 * 10**6, 180 * 10**6):
        mine = vg.primes.in_range_with_limit(a, a + width, 2 * 10**7)
        assert mine == oracle_lib.primes_in_range(a, a + width).tolist(), (a, width)


PROBE = r"""
#include <cstdio>
#include "engine.h"
using namespace vg;

int main() {
  int runs = 0;
  auto failing = [&](int times, int code) {
    runs = 0;
    return [&runs, times, code] { if (runs++ < times) throw Error(code, "no room"); return 7; };
  };
  auto go = [&](bool held, int times, int code) {
    std::shared_ptr<int> kept = held ? std::make_shared<int>(1) : nullptr;
    int rc = 0;
    try { rc = with_room(kept, failing(times, code)); } catch (const Error& e) { rc = -e.code; }
    std::printf("%d %d %d\n", rc, runs, kept ? 1 : 0);
  };
  go(true, 0, 0);                          // nothing failed: the buffers stay
  go(true, 1, VOSS_ERR_OUT_OF_MEMORY);     // again without them
  go(true, 2, VOSS_ERR_OUT_OF_MEMORY);     // once only
  go(false, 1, VOSS_ERR_OUT_OF_MEMORY);    // nothing to give back
  go(true, 1, VOSS_ERR_CUDA);              // another error
  return 0;
}
"""


def test_out_of_memory_gives_kept_buffers_back(tmp_path):
    gxx, cuda = shutil.which("g++"), os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include"
    if not gxx or not os.path.exists(cuda + "/cuda_runtime.h"):
        pytest.skip("no g++ or CUDA headers")
    (tmp_path / "probe.cpp").write_text(PROBE)
    exe = tmp_path / "probe"
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", str(ROOT / "voss_gb300" / "csrc"), "-I", str(ROOT / "include"),
                    "-I", cuda, str(tmp_path / "probe.cpp"), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()
    assert out == ["7 1 1", "7 2 0", "-4 2 0", "-4 1 0", "-5 1 1"]
