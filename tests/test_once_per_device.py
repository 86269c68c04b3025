"""Kernel attributes are set once for every device, not once for the process: the
helper that every launch with dynamic shared memory goes through runs its set-up
for each device that launches, again after a failure, and never twice after a
success, from several threads too."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "salvus_b200", "csrc")

PROGRAM = r"""
#include "once_per_device.h"
#include <cstdio>
#include <thread>
#include <vector>
#define CHECK(x) if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; }
int main() {
  salvus::OncePerDevice once;
  std::vector<int> calls;
  auto set = [&](int device, int rc) { return once(device, [&] { calls.push_back(device); return rc; }); };
  CHECK(set(0, 0) == 0 && set(0, 0) == 0 && calls == std::vector<int>({0}));
  CHECK(set(1, 0) == 0 && calls.back() == 1 && calls.size() == 2);
  CHECK(set(63, 7) == 7 && calls.back() == 63);
  CHECK(set(63, 0) == 0 && calls.size() == 4 && set(63, 0) == 0 && calls.size() == 4);
  CHECK(set(64, 0) == 0 && set(64, 0) == 0 && calls.size() == 6);
  CHECK(set(0, 0) == 0 && set(1, 0) == 0 && calls.size() == 6);
  salvus::OncePerDevice shared;
  std::atomic<int> n{0};
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&, t] {
      for (int k = 0; k < 1000; ++k) shared(t % 4, [&] { ++n; return 0; });
    });
  for (auto &t : threads) t.join();
  CHECK(n >= 4 && n <= 8);
  std::puts("ok");
}
"""


def test_set_up_runs_once_per_device(tmp_path):
    src = tmp_path / "once.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "once")
    subprocess.check_call(["g++", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", exe])
    assert subprocess.run([exe], capture_output=True, text=True).stdout == "ok\n"


def test_no_process_wide_flag_guards_an_attribute():
    with open(os.path.join(CSRC, "abi.cu")) as f:
        text = f.read()
    for at in re.finditer("cudaFuncSetAttribute", text):
        assert "static bool" not in text[at.start() - 200:at.start()]
