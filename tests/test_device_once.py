"""Set-up once per device and key (csrc/device_once.h, which raises the kernels' shared-memory limits): a second
device gets its own, a failure is tried again, threads that come together run it once (host C++, no GPU); and no
source keeps a process-wide flag for it."""
import glob
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "femflow_gb300", "csrc")

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "device_once.h"
int main() {
  ffmpm::DeviceOnce once;
  int a = 0, b = 0, calls = 0;
  auto ok = [&] { ++calls; return true; };
  auto fail = [&] { ++calls; return false; };
  bool r = once.run(0, &a, ok) && once.run(0, &a, ok) && calls == 1;  // once
  r = r && once.run(1, &a, ok) && calls == 2;                          // another device
  r = r && once.run(0, &b, ok) && calls == 3;                          // another key
  r = r && !once.run(2, &a, fail) && !once.run(2, &a, fail) && calls == 5 && once.run(2, &a, ok) && calls == 6;
  std::atomic<int> n{0};
  std::vector<std::thread> t;
  for (int i = 0; i < 8; ++i) t.emplace_back([&] { once.run(3, &a, [&] { ++n; return true; }); });
  for (auto& x : t) x.join();
  printf("%d\n", r && n == 1);
}
"""


def test_once_per_device_and_key(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.strip() == "1"


def test_kernel_attributes_are_set_per_device_or_on_every_call():
    for f in glob.glob(os.path.join(CSRC, "*.cu")):
        assert not re.search(r"static\s+bool\s+\w+\s*=\s*false", open(f).read()), f
