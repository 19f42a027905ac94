"""The guard that sets the kernels' shared-memory limits once per device
(csrc/device_once.h), compiled for the host: every device gets its own call,
an error is returned and left to the next caller, and threads that arrive
together wait for the one that does the work."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "matched-time-splitting-3d_b200", "csrc")
PROGRAM = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>

#include "device_once.h"

#define CHECK(x) if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; }

int main() {
  mts::DeviceOnce once;
  int calls[66] = {};
  auto work = [&](int device, int error) { return once.run(device, [&] { calls[device]++; return error; }); };
  CHECK(work(0, 0) == 0 && work(0, 0) == 0 && calls[0] == 1);
  CHECK(work(1, 7) == 7 && calls[1] == 1);              // an error: returned, not remembered
  CHECK(work(1, 0) == 0 && work(1, 0) == 0 && calls[1] == 2);
  CHECK(work(63, 0) == 0 && work(63, 0) == 0 && calls[63] == 1);
  CHECK(work(65, 0) == 0 && work(65, 0) == 0 && calls[65] == 2);  // past the mask: every time

  mts::DeviceOnce shared;
  std::atomic<int> done{0}, early{0}, made{0};
  std::vector<std::thread> ts;
  for (int i = 0; i < 16; i++)
    ts.emplace_back([&] {
      shared.run(3, [&] {
        std::this_thread::sleep_for(std::chrono::milliseconds(50));
        made++;
        done = 1;
        return 0;
      });
      if (!done) early++;
    });
  for (auto& t : ts) t.join();
  CHECK(made == 1 && early == 0);
  return 0;
}
"""


def test_each_device_once(tmp_path):
    src = tmp_path / "once.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "once"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    cp = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert cp.returncode == 0, cp.stdout


def test_no_limit_is_set_behind_a_process_wide_flag():
    """Every call that sets a limit goes through the guard: none is made at
    handle creation for all kernels, and no return code is dropped."""
    with open(os.path.join(CSRC, "capi.cu")) as f:
        capi = f.read()
    assert "static bool" not in capi
    for name in os.listdir(CSRC):
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        calls = text.count("cudaFuncSetAttribute(")
        assert calls == (1 if name == "device_common.cuh" else 0), name
