"""Kernel attributes are set on every device that launches the kernel (csrc/device_limits.h), checked on the host."""
import os
import shutil
import subprocess

import pytest

from conftest import REPO

SRC = r"""
#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>
#include "device_limits.h"

int main() {
  impes::DeviceLimits d;
  int a = 0, b = 0, calls = 0;
  auto set = [&](size_t) { ++calls; };
  d.raise(0, &a, 100, set);                 // set
  d.raise(0, &a, 100, set);                 // held
  d.raise(0, &a, 60, set);                  // lower: held
  if (calls != 1) return 1;
  d.raise(1, &a, 100, set);                 // another device: set there too
  if (calls != 2) return 2;
  d.raise(1, &a, 60, set);
  d.raise(0, &b, 60, set);                  // another kernel
  if (calls != 3) return 3;
  d.raise(0, &a, 200, set);                 // higher: set again, on this device alone
  d.raise(1, &a, 200, set);
  if (calls != 5) return 4;
  try {                                     // a refused value is not held
    d.raise(2, &a, 10, [](size_t) { throw std::runtime_error("refused"); });
    return 5;
  } catch (const std::runtime_error&) {
  }
  d.raise(2, &a, 10, set);
  if (calls != 6) return 6;
  int most = 0;                             // from several threads: the largest is set last
  std::vector<std::thread> t;
  for (int q = 1; q <= 8; ++q)
    t.emplace_back([&, q] { d.raise(3, &a, 10 * q, [&](size_t v) { most = (int)v; }); });
  for (auto& x : t) x.join();
  return most == 80 ? 0 : 7;
}
"""


def test_attributes_are_held_per_device(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "limits.cpp", tmp_path / "limits"
    src.write_text(SRC)
    inc = os.path.join(REPO, "oil-simulator-py_b200", "csrc")
    subprocess.run([gxx, "-std=c++17", "-Wall", "-Werror", "-pthread", "-I", inc, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_attribute_is_set_once_per_process():
    """A function-local static runs once in the process, whatever device is current."""
    csrc = os.path.join(REPO, "oil-simulator-py_b200", "csrc")
    for name in sorted(os.listdir(csrc)):
        if not name.endswith((".cu", ".cuh", ".h")):
            continue
        with open(os.path.join(csrc, name)) as f:
            for stmt in f.read().split(";"):
                assert not ("static" in stmt and "cudaFuncSetAttribute" in stmt), (name, stmt)
