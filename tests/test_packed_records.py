"""Packed records that an update wrote for the next pass (csrc/packed_records.h) serve that
pass of the same call and no other, also after an error: on the host compiler."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "flowunsteady_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "packed_records.h"

static vpm::PackedRecords packed;
static int bad = 0;
static void expect(bool got, bool want, int line) {
  if (got != want) std::printf("line %d\n", line), ++bad;
}
#define EXPECT(got, want) expect(got, want, __LINE__)

// A call of three passes, each leaving records for the next; pass `fail` fails.
static int call(int fail) {
  const vpm::PackedRecords::Scope scope(packed);
  for (int pass = 0; pass < 3; ++pass) {
    EXPECT(packed.take(pass, 1.0), pass > 0);
    if (pass == fail) return 1;
    packed.hold(pass + 1, 1.0);
    if (pass + 10 == fail) return 1;   // fails once its records are written
  }
  return 0;
}

int main() {
  EXPECT(packed.take(0, 1.0), false);
  packed.hold(2, 0.5);
  EXPECT(packed.take(2, 1.0), false);   // another scale
  EXPECT(packed.take(2, 0.5), false);   // and dropped by the pass in between
  packed.hold(2, 0.5);
  EXPECT(packed.take(1, 0.5), false);   // another pass
  packed.hold(2, 0.5);
  EXPECT(packed.take(2, 0.5), true);
  EXPECT(packed.take(2, 0.5), false);   // once
  packed.hold(-1, 1.0);
  EXPECT(packed.take(-1, 1.0), false);
  for (int fail : {-1, 0, 1, 2, 10, 11, 12})
    for (int pass = 0; pass < 4; ++pass) {
      call(fail);
      EXPECT(packed.take(pass, 1.0), false);
    }
  std::printf("%d\n", bad);
  return bad;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_records_serve_one_pass_of_one_call(tmp_path):
    src, exe = tmp_path / "packed.cpp", tmp_path / "packed"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.stdout.strip() == "0"
