"""Shared-memory limits of kernels: the once-per-device registry, compiled and
run on the host, and that no launch sets a limit of its own size (the limit is
shared by all threads, so a smaller call would lower it under a larger one)."""
import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fastpls_b200", "csrc")

PROGRAM = r"""
#include "once_per_device.hpp"
#include <atomic>
#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>

int main() {
  fpls::OncePerDevice once;
  static int keys[3];
  std::atomic<int> calls[3][4] = {}, seen_before_run{0};
  std::atomic<bool> ready[3][4] = {};
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&, t] {
      for (int r = 0; r < 2000; ++r) {
        const int k = (r + t) % 3, d = (r / 3 + t) % 4;
        once.run(&keys[k], d, [&] {
          calls[k][d]++;
          std::this_thread::yield();
          ready[k][d] = true;
        });
        if (!ready[k][d]) seen_before_run++;  // returned before the first run had finished
      }
    });
  for (auto& t : threads) t.join();
  for (auto& row : calls)
    for (auto& c : row)
      if (c != 1) return 1;
  if (seen_before_run) return 2;
  int tries = 0;
  for (int r = 0; r < 3; ++r) {
    try {
      once.run(&tries, 0, [&] { if (++tries < 2) throw std::runtime_error("refused"); });
    } catch (const std::runtime_error&) {
    }
  }
  return tries == 2 ? 0 : 3;
}
"""


def test_once_per_key_and_device(tmp_path):
    src = tmp_path / "once.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "once"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0


def test_no_limit_follows_a_call():
    """Every limit is a constant or the device's: none names a size computed
    for the call."""
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        text = open(path).read()
        for m in re.finditer(r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*\(int\)\s*smem_?\w*\b", text):
            line = text[:m.start()].count("\n") + 1
            # a size that is a constant of the kernel's template
            assert "constexpr size_t smem" in text, f"{os.path.basename(path)}:{line}"


def test_every_limit_is_set_per_device():
    """The limit belongs to one device: only the registry sets it, so a thread
    on another device of the process gets it too."""
    sites = []
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        text = open(path).read()
        for m in re.finditer(r"cudaFuncSetAttribute\(", text):
            body = text[:m.start()].rsplit("\n}", 1)[-1]
            if "void allow_shared_memory(const void* kernel) {" not in body:
                sites.append(f"{os.path.basename(path)}:{text[:m.start()].count(chr(10)) + 1}")
    assert not sites, sites
