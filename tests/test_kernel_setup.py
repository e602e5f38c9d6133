"""First-use set-up of the kernels, compiled for the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "once.h"
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>

int main() {
  orinfer::OncePerSlot<2, 4> once;
  // a failure is returned and the next caller tries again
  int calls = 0;
  if (once.run(0, 1, [&] { ++calls; return 7; }) != 7) return 1;
  if (once.run(0, 1, [&] { ++calls; return 0; }) != 0 || calls != 2) return 2;
  if (once.run(0, 1, [&] { ++calls; return 9; }) != 0 || calls != 2) return 3;
  // per device and per slot
  if (once.run(1, 1, [&] { ++calls; return 0; }) != 0 || calls != 3) return 4;
  if (once.run(0, 2, [&] { ++calls; return 0; }) != 0 || calls != 4) return 5;
  // nothing is remembered outside the table
  for (int slot : {-1, 4})
    for (int i = 0; i < 2; ++i)
      if (once.run(0, slot, [] { return 3; }) != 3) return 6;
  if (once.run(-1, 0, [] { return 3; }) != 3 || once.run(2, 0, [] { return 3; }) != 3) return 7;
  // no thread is past the set-up before it is through
  for (int round = 0; round < 20; ++round) {
    orinfer::OncePerSlot<1, 1> fresh;
    std::atomic<int> set{0}, runs{0}, early{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
      threads.emplace_back([&] {
        const int r = fresh.run(0, 0, [&] {
          ++runs;
          std::this_thread::sleep_for(std::chrono::milliseconds(5));
          set = 1;
          return 0;
        });
        if (r != 0 || set != 1) ++early;
      });
    for (auto& t : threads) t.join();
    if (early != 0 || runs != 1) return 8;
  }
  std::puts("ok");
  return 0;
}
"""


def test_set_up_runs_once_and_before_anyone_passes(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I",
                    os.path.join(ROOT, "csrc", "kernels"), str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.returncode
