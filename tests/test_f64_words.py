"""Tests on the words of FP64 numbers that bound reads of the FP64 tables
(csrc/f64_tables.cuh), compiled for the host."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "flowunsteady_gb300", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include "f64_tables.cuh"

static double value(uint32_t hi, uint32_t lo) {
  const uint64_t b = uint64_t(hi) << 32 | lo;
  double d;
  std::memcpy(&d, &b, 8);
  return d;
}

int main() {
  // Every high word on a coarse walk, and around the ends: what counts as near has its
  // row inside the table, as core_f12 forms it; what is not in [0, 45) is far.
  long bad = 0;
  auto check = [&](uint32_t hi) {
    for (uint32_t lo : {0u, 1u, 0x7fffffffu, 0x80000000u, 0xffffffffu}) {
      const double u = value(hi, lo);
      const bool near = vpm::core_near_word(hi);
      if (near != (u >= 0.0 && u < 45.0 && !std::signbit(u))) ++bad;
      if (!near) continue;
      const double t = std::fma(u, 16.0, 6755399441055744.0);
      uint64_t b;
      std::memcpy(&b, &t, 8);
      const int32_t row = int32_t(uint32_t(b));
      if (row < 0 || row >= vpm::kCoreRows) ++bad;
    }
  };
  for (uint64_t hi = 0; hi <= 0xffffffffull; hi += 4093) check(uint32_t(hi));
  for (uint32_t mid : {0u, 0x3ff00000u, 0x40468000u, 0x7ff00000u, 0x7ff80000u, 0x80000000u,
                       0xfff00000u, 0xfff80000u})
    for (int d = -64; d <= 64; ++d) check(mid + uint32_t(d));
  std::printf("%ld\n", bad);
  return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_only_words_of_the_core_table_count_as_near(tmp_path):
    src, exe = tmp_path / "words.cpp", tmp_path / "words"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)])
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout.strip() == "0"
