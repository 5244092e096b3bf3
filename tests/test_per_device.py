"""PerDevice (per_device.hpp), which holds the kernels' attributes and occupancies: made once for each
device however many threads ask, again after a call that threw, an index past its size refused. On the
host: a small program against the header."""
import shutil
import subprocess

import pytest

SOURCE = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include "per_device.hpp"
int main() {
  static fx::PerDevice<int> known;
  std::atomic<int> made[2] = {{0}, {0}};
  std::vector<std::thread> threads;
  std::atomic<int> wrong{0};
  for (int t = 0; t < 16; ++t)
    threads.emplace_back([&, t] {
      for (int i = 0; i < 1000; ++i) {
        const int dev = (t + i) % 2;
        const int got = known.get(dev, [&] { return 10 + dev + 0 * ++made[dev]; });
        if (got != 10 + dev) ++wrong;
      }
    });
  for (auto& t : threads) t.join();
  fx::PerDevice<int> later;
  int refused = 0, calls = 0;
  for (int i = 0; i < 2; ++i) try {
      later.get(3, [&]() -> int { if (++calls == 1) throw fx::Error(FX_E_CUDA, "first"); return 7; });
    } catch (const fx::Error&) { ++refused; }
  const int third = later.get(3, [&] { ++calls; return 8; });
  int past = 0;
  for (int dev : {-1, fx::kMaxDevices}) try { later.get(dev, [] { return 1; }); } catch (const fx::Error& e) { past += e.code; }
  std::printf("%d %d %d %d %d %d %d\n", made[0].load(), made[1].load(), wrong.load(), refused, calls, third, past);
}
"""


def test_once_per_device(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    from femorax_b200.build import CSRC
    src, exe = tmp_path / "per_device.cpp", tmp_path / "per_device"
    src.write_text(SOURCE)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe), "-lpthread"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True, timeout=60).stdout.split()
    assert out == ["1", "1", "0", "1", "2", "7", "4"]  # past: twice FX_E_UNSUPPORTED
