"""Launch settings are found for every device of the process, not once for the
process: a kernel opted in to more shared memory on the first device only could
not be launched on the second."""
import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "vitrum_b200", "csrc")

PROGRAM = r"""
#include <atomic>
#include <cassert>
#include <stdexcept>
#include <thread>
#include <vector>
#include "per_device.h"

int main() {
  vt::PerDevice<int> p;
  std::atomic<int> found[4] = {};
  auto ask = [&](int device) { return p.get(device, [&, device] { ++found[device]; return 10 + device; }); };
  bool threw = false;
  try {
    p.get(3, []() -> int { throw std::runtime_error("no such attribute"); });
  } catch (const std::runtime_error&) {
    threw = true;
  }
  assert(threw);
  std::vector<std::thread> threads;
  std::atomic<int> wrong{0};
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&] {
      for (int i = 0; i < 1000; ++i)
        for (int device = 0; device < 4; ++device) wrong += ask(device) != 10 + device;
    });
  for (auto& t : threads) t.join();
  assert(wrong == 0);
  for (auto& f : found) assert(f == 1);
  int calls = 0;
  for (int i = 0; i < 2; ++i) assert(p.get(1000, [&] { return ++calls; }) == calls);
  assert(calls == 2);
  return 0;
}
"""


def test_found_once_for_each_device(tmp_path):
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)


def test_no_launch_setting_is_kept_for_the_process():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = open(path).read()
        for m in re.finditer(r"cudaFuncSetAttribute|cudaOccupancyMax|MemPoolSetAttribute", text):
            before = text[max(0, m.start() - 400):m.start()]
            assert not re.search(r"static (bool|int|size_t)\s+\w+(\[\w*\])?\s*=", before), (path, m.group())
