"""A kernel's attributes are set in every device context it runs in (csrc/per_context.h),
with the CUDA calls replaced by a count, on the host compiler."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "flowunsteady_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include <thread>
#include <vector>
#include "per_context.h"

int main() {
  int calls = 0, result = 0, bad = 0;
  vpm::PerContext done;
  auto set = [&] { ++calls; return result; };
  auto expect = [&](int dev, unsigned long long ctx, int rc, int n) {
    calls = 0;
    if (done.ensure(dev, ctx, set) != rc || calls != n) {
      ++bad;
      std::printf("device %d context %llu: %d calls\n", dev, ctx, calls);
    }
  };
  expect(0, 11, 0, 1);   // the first call on a device
  expect(0, 11, 0, 0);
  expect(1, 12, 0, 1);   // another device
  expect(1, 12, 0, 0);
  expect(0, 11, 0, 0);   // and back
  expect(0, 13, 0, 1);   // the first device's context replaced
  expect(0, 13, 0, 0);
  expect(63, 14, 0, 1);
  expect(63, 14, 0, 0);
  for (int dev : {64, 1000, -1}) {   // beyond the table, and unknown contexts: every time
    expect(dev, 15, 0, 1);
    expect(dev, 15, 0, 1);
  }
  expect(2, 0, 0, 1);
  expect(2, 0, 0, 1);
  result = 7;            // a failure is returned and tried again
  expect(2, 16, 7, 1);
  expect(2, 16, 7, 1);
  result = 0;
  expect(2, 16, 0, 1);
  expect(2, 16, 0, 0);
  vpm::PerContext shared;   // threads on several devices: set before any of them goes on
  std::vector<std::thread> ts;
  std::atomic<int> ok{0};
  for (int t = 0; t < 8; ++t)
    ts.emplace_back([&, t] {
      thread_local int mine = 0;
      shared.ensure(t % 4, 100 + t % 4, [&] { return mine = 1, 0; });
      ok += shared.ensure(t % 4, 100 + t % 4, [] { return 1; }) == 0;
    });
  for (auto& t : ts) t.join();
  bad += ok != 8;
  std::printf("%d\n", bad);
  return bad;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_set_up_runs_once_in_every_context(tmp_path):
    src, exe = tmp_path / "per_context.cpp", tmp_path / "per_context"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.stdout.strip() == "0"
