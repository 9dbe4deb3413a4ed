"""The fixed-point phase sum of the float64 kernels (``wide_mac`` and ``wide_fraction``
of csrc/gwl_wide.cuh) on the host: the value modulo one cycle of coefficients and
table entries at the ends of their ranges, with the compiler's check of signed
overflow on, against 128-bit integers."""
import os
import subprocess

import pytest

from bilby_gb300 import _build
from tests.conftest import ROOT

PROBE = r"""
#include <cstdio>
#include <cstdlib>
#include "gwl_wide.cuh"
int main() {
  // coefficients c = ch 2^27 + cl of 59 bits, table entries m = mh 2^27 + ml of 58
  const int64_t cs[] = {((int64_t)1 << 58) - 1, -((int64_t)1 << 58), ((int64_t)1 << 57) + 12345, -987654321987, 0};
  const int64_t ms[] = {((int64_t)1 << 58) - 1, ((int64_t)1 << 57) + 1, 123456789123456789, 1, 0};
  unsigned seed = 1;
  for (int round = 0; round < 2000; ++round) {
    uint64_t acc = 0;
    int64_t cross = 0;
    __int128 exact = 0;
    for (int b = 0; b < gwl::kNumBasis; ++b) {
      const int64_t c = round == 0 ? cs[0] : round == 1 ? cs[1] : cs[(seed = seed * 1103515245u + 12345u) / 65536u % 5];
      const int64_t m = round < 2 ? ms[0] : ms[(seed = seed * 1103515245u + 12345u) / 65536u % 5];
      gwl::wide_mac(acc, cross, (int32_t)(c >> 27), (int32_t)(c & 0x7ffffff), (int32_t)(m & 0x7ffffff), (int32_t)(m >> 27));
      exact += (__int128)c * m;
    }
    // c 2^(s - 58) times m 2^-58 cycles: the fraction in units of 2^-64 is exact 2^(s - 52)
    const int s = 14;
    const uint64_t got = gwl::wide_fraction(acc, cross, s + 2), want = (uint64_t)(exact >> (52 - s));
    const int64_t off = (int64_t)(want - got);  // the low products dropped: 8 of 2^54, and a rounding
    if (off < -1 || off > ((int64_t)9 << (s + 2))) {
      std::printf("round %d: %llx for %llx\n", round, (unsigned long long)got, (unsigned long long)want);
      return 1;
    }
  }
  std::printf("same");
}
"""


def test_phase_sum_at_the_ends_of_its_range(tmp_path):
    (tmp_path / "probe.cu").write_text(PROBE)
    exe = tmp_path / "probe"
    cmd = [_build.nvcc(), *_build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "bilby_gb300", "csrc"),
           "-I", os.path.join(ROOT, "include"), "-Xcompiler",
           "-fsanitize=signed-integer-overflow", "-Xcompiler", "-fno-sanitize-recover=all", str(tmp_path / "probe.cu"), "-o", str(exe)]
    built = subprocess.run(cmd, capture_output=True, text=True)
    if built.returncode != 0 and "ubsan" in built.stderr:
        pytest.skip("no undefined-behaviour sanitizer")
    assert built.returncode == 0, built.stderr
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout == "same", res.stdout + res.stderr
