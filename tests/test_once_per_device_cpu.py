"""Work that each device of a process needs once (csrc/once_per_device.h): done on every device, again after a
failure, by one of the threads that ask for it at the same time, and nowhere when there is no such device."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cassert>
#include <chrono>
#include <thread>
#include <vector>
#include "once_per_device.h"

int main() {
  mw::OncePerDevice a, b;
  int calls[64] = {};
  auto work = [&](int dev, bool ok) { return [&calls, dev, ok] { ++calls[dev]; return ok; }; };
  for (int round = 0; round < 3; ++round)
    for (int dev : {0, 1, 7, 63}) assert(a.run(dev, work(dev, true)));
  for (int dev : {0, 1, 7, 63}) assert(calls[dev] == 1);
  assert(!a.run(2, work(2, false)) && !a.run(2, work(2, false)) && a.run(2, work(2, true)) && a.run(2, work(2, true)));
  assert(calls[2] == 3);
  assert(!a.run(-1, [] { assert(false); return true; }) && !a.run(64, [] { assert(false); return true; }));
  assert(b.run(0, work(0, true)) && calls[0] == 2);
  std::atomic<int> done{0}, started{0};
  std::vector<std::thread> pool;
  for (int t = 0; t < 8; ++t)
    pool.emplace_back([&] {
      assert(b.run(5, [&] {
        ++started;
        std::this_thread::sleep_for(std::chrono::milliseconds(20));
        done = 1;
        return true;
      }));
      assert(done == 1);
    });
  for (auto& t : pool) t.join();
  assert(started == 1);
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "meeuuw_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True, timeout=120)
    subprocess.run([str(exe)], check=True, timeout=60)


def test_no_process_wide_flags():
    """What is set up per device is not remembered by a plain static flag."""
    csrc = os.path.join(ROOT, "meeuuw_b200", "csrc")
    for name in sorted(os.listdir(csrc)):
        for line in open(os.path.join(csrc, name)):
            assert not line.strip().startswith(("static bool attr", "static bool ready", "static size_t attr")), (name, line)
