"""Attributes that belong to a device are set on each device of a process (csrc/common/per_device.h), on the host alone."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oneflow_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "common/per_device.h"
int main() {
  ofb::OncePerDevice once;
  int calls[80] = {0};
  auto ok = [&](int d) { return once(d, [&] { ++calls[d]; return 0; }); };
  for (int round = 0; round < 3; ++round)
    for (int d = 0; d < 4; ++d) if (ok(d)) return 1;
  for (int d = 0; d < 4; ++d) if (calls[d] != 1) return 2;          // once each, and not only on the first device
  int tries = 0;
  if (once(7, [&] { ++tries; return 5; }) != 5) return 3;           // a failure is reported and tried again
  if (once(7, [&] { ++tries; return 0; }) != 0 || tries != 2) return 4;
  for (int round = 0; round < 2; ++round) if (ok(63) || ok(64)) return 5;
  if (calls[63] != 1 || calls[64] != 2) return 6;
  ofb::OncePerDevice shared;
  std::vector<std::thread> threads;
  std::atomic<int> set{0};
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&] { for (int d = 0; d < 8; ++d) shared(d, [&] { ++set; return 0; }); });
  for (auto& t : threads) t.join();
  if (set < 8) return 7;
  const int before = set;
  for (int d = 0; d < 8; ++d) shared(d, [&] { ++set; return 0; });
  return set == before ? 0 : 8;
}
"""


def test_once_per_device(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "per_device.cpp", tmp_path / "per_device"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_launcher_sets_an_attribute_once_per_process():
    for folder, _, files in os.walk(CSRC):
        for name in files:
            if name.endswith((".cu", ".cuh", ".cpp", ".h")):
                for number, line in enumerate(open(os.path.join(folder, name)), 1):
                    if "cudaFuncSetAttribute(" in line and not line.lstrip().startswith("//"):
                        assert "OFB_CUDA_OK_ONCE_PER_DEVICE(" in line, f"{name}:{number}"
