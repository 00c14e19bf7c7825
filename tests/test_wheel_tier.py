"""The wheel tier: its host-built table (CPU) and its marking (GPU) where it can
go wrong -- segments that hold their own sieving primes, primes just below and
above the segment and 2.5 segments, partial rows and units, short last
segments."""
import subprocess

import numpy as np
import pytest

from conftest import ROOT

W30 = (1, 7, 11, 13, 17, 19, 23, 29)

PROBE = r"""
#define __host__
#define __device__
#include <cstdio>
#include <vector>
#include "sieve.cuh"
int main(int, char** argv) {
  std::vector<uint32_t> P;
  for (uint32_t c = vg::kFirstTablePrime; c < (uint32_t)atoi(argv[1]); ++c) {
    bool prime = true;
    for (uint32_t d = 2; d * d <= c && prime; ++d) prime = c % d != 0;
    if (prime) P.push_back(c);
  }
  const uint32_t n = (uint32_t)P.size();
  std::vector<vg::WheelEntry> W(n + 1);
  std::vector<uint32_t> off(8 * vg::wheel_rows(n));
  vg::build_wheel_table(P.data(), n, W.data(), off.data());
  for (uint32_t i = 0; i < n; ++i) std::printf("e %u %u\n", W[i].t, W[i].inv);
  for (uint32_t r = 0; r < vg::wheel_rows(n); ++r) {
    std::printf("r");
    for (int k = 0; k < 8; ++k) std::printf(" %u", off[8 * r + k]);
    std::printf("\n");
  }
  const vg::WheelClasses C = vg::make_wheel_classes();
  for (int k = 0; k < 8; ++k)
    for (int j = 0; j < 8; ++j)
      std::printf("c %d %d %u %u %u\n", k, j, C.c[k].step[j], ~C.c[k].keep[j], C.c[k].bstep[j]);
  return 0;
}
"""


@pytest.mark.parametrize("limit", [62, 67, 1031, 5000, 30011])
def test_wheel_table(tmp_path, limit):
    src = tmp_path / "probe.cpp"
    src.write_text("#include <cstdlib>\n" + PROBE)
    exe = tmp_path / "probe"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "voss_gb300" / "csrc"), str(src), "-o", str(exe)],
                   check=True)
    lines = [l.split() for l in subprocess.run([str(exe), str(limit)], check=True, capture_output=True,
                                               text=True).stdout.splitlines()]
    primes = [c for c in range(61, limit) if all(c % d for d in range(2, int(c ** 0.5) + 1))]
    want = [p for c in W30 for p in primes if p % 30 == c]
    entries = [(int(t), int(inv)) for k, t, inv in (l for l in lines if l[0] == "e")]
    assert [t for t, _ in entries] == [p // 30 for p in want]
    assert [inv for _, inv in entries] == [(1 << 42) // p if p > 1024 else 0 for p in want]
    rows = [list(map(int, l[1:])) for l in lines if l[0] == "r"]
    assert len(rows) == len(primes) // 64 + 2
    for r, row in enumerate(rows):
        below = primes[:64 * r]
        for k, c in enumerate(W30):
            start = sum(p % 30 in W30[:k] for p in primes)
            assert row[k] == start + sum(p % 30 == c for p in below), (r, k)
    # the class constants give every multiple's byte and bit: p (30 a + w) for p = 30 t + c
    for k, c in enumerate(W30):
        byte, index = 0, 0
        for _, kk, j, step, bit, bstep in (l for l in lines if l[0] == "c" and int(l[1]) == k):
            w = W30[int(j)]
            byte += int(step)
            index = (index + int(bstep)) % (1 << 32)
            o = W30.index(c * w % 30)
            assert byte == c * w // 30 and int(bit) == 1 << o and index == 8 * byte + o, (c, w)


@pytest.mark.gpu
@pytest.mark.parametrize("seg_bytes", [1024, 4096, 16384, 65536, 222848])
def test_wheel_tier_vs_oracle(vg, oracle_lib, seg_bytes):
    base = vg.primes.get_config()
    try:
        vg.primes.set_config(seg_bytes=seg_bytes, threads=1024, tier_split=512, bucket_split=0, auto_tune=0)
        span = 30 * seg_bytes
        cases = [(0, 3 * span + 1), (1, 2600), (2579, 2 * span + 17), (3839, 3841 + span), (30 * 127, 30 * 129 + span),
                 (span - 1, span + 1),
                 # p*p just below and above the end, for p near the segment and 2.5 segments
                 *(((p * p - span) // 7 * 7, p * p + d) for p in (seg_bytes, 5 * seg_bytes // 2) if p * p > span
                   for d in (-2, 3)),
                 (10**12 - 12345, 10**12 - 12345 + 2 * span + 31), (10**14 + 10**10 - span, 10**14 + 10**10 + 1)]
        for a, b in cases:
            st, orc = vg.range_stats(a, b, full=True), oracle_lib.range_stats(a, b)
            for k in ("count", "pi_4_1", "pi_4_3", "pi_3_1", "pi_3_2", "max_gap", "max_gap_start", "num_gaps"):
                assert getattr(st, k) == orc[k], (a, b, k)
            assert (st.first_prime, st.last_prime) == (orc["first"], orc["last"]), (a, b)
            assert np.array_equal(np.array(st.gap_hist_full, dtype=np.uint64), orc["hist"]), (a, b)
    finally:
        vg.primes.set_config(**base)
