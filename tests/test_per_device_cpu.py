"""Kernels are set up once on every device of the process, from any thread."""
import glob
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(__file__), "..", "capytaine_b200", "csrc")

PROGRAM = r"""
#include <cassert>
#include <thread>
#include <vector>
#include "per_device.h"
int main() {
  static bem::OncePerDevice once;
  std::atomic<int> calls[3] = {};
  auto use = [&](int dev) { return once(dev, [&] { ++calls[dev]; return 0; }); };
  for (int i = 0; i < 5; ++i)
    for (int dev = 0; dev < 2; ++dev) assert(use(dev) == 0);
  assert(calls[0] == 1 && calls[1] == 1);
  // a failed set-up is reported and tried again
  assert(once(2, [] { return 7; }) == 7 && use(2) == 0 && calls[2] == 1);
  // indices without an entry: every time
  int n = 0;
  for (int dev : {-1, 64, 64, 1000}) once(dev, [&] { ++n; return 0; });
  assert(n == 4);
  // threads: nobody goes on before a set-up of the device has returned
  static bem::OncePerDevice shared;
  std::atomic<bool> ready[8] = {};
  std::vector<std::thread> threads;
  for (int t = 0; t < 16; ++t)
    threads.emplace_back([&, t] {
      shared(t % 8, [&] { ready[t % 8] = true; return 0; });
      assert(ready[t % 8]);
    });
  for (auto& t : threads) t.join();
}
"""


def test_once_per_device(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", CSRC, "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")],
                   check=True)
    subprocess.run([str(tmp_path / "t")], check=True)


def test_every_shared_memory_opt_in_is_per_device():
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = open(path).read()
        assert not re.search(r"\bbool\s+\w*configured\b", text), path
        if "cudaFuncAttributeMaxDynamicSharedMemorySize" in text and not path.endswith("noalloc.cu"):
            assert "OncePerDevice" in text, path
