"""parallel_for (engine.cuh), compiled alone: every index once, and an exception
of the body, on whichever thread, reaches the caller as that exception."""
import subprocess

SRC = r"""
#include <cstdio>
#include <new>
#include "engine.cuh"

int main() {
  for (uint64_t n : {0, 1, 2, 63, 64, 65, 5000}) {
    std::vector<std::atomic<int>> seen(n);
    bf::parallel_for(n, [&](uint64_t i) { ++seen[i]; });
    for (auto& s : seen)
      if (s != 1) return 1;
    for (uint64_t bad : {uint64_t(0), n / 2, n - 1}) {
      if (!n) continue;
      bool caught = false;
      try {
        bf::parallel_for(n, [&](uint64_t i) {
          if (i >= bad) throw std::bad_alloc();
        });
      } catch (const std::bad_alloc&) {
        caught = true;
      }
      if (!caught) return 2;
    }
  }
  std::puts("ok");
}
"""


def test_parallel_for(tmp_path):
    import build
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run([build.NVCC, "-std=c++17", "-I", str(build.PKG / "csrc"), "-I",
                    str(build.ROOT / "include"), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r
