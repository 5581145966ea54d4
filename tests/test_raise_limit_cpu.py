"""Two host threads that raise one kernel's shared-memory limit at once: the larger
value stays, in whatever order they read and write it."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "ionosphere_fdtd_b200" / "csrc"

PROGRAM = r"""
#include <chrono>
#include <cstdio>
#include <thread>
#include "raise_limit.h"
static size_t limit = 0;
static void nap(int ms) { std::this_thread::sleep_for(std::chrono::milliseconds(ms)); }
static int raise(size_t bytes, int before_read, int before_write) {
  nap(before_read);
  return ifdtd::raise_limit(
      bytes, [&](size_t* now) { *now = limit; nap(before_write); return 0; }, [&](size_t b) { limit = b; return 0; });
}
int main() {
  // the thread that needs less reads first and writes last
  std::thread less([] { raise(100, 0, 60); }), more([] { raise(200, 20, 0); });
  less.join();
  more.join();
  const size_t after = limit;
  const int refused = ifdtd::raise_limit(300, [](size_t*) { return 7; }, [](size_t) { return 0; });
  std::printf("%zu %d %zu\n", after, refused, limit);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_the_larger_limit_stays(tmp_path):
    (tmp_path / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", str(CSRC), "-o", str(tmp_path / "main"), str(tmp_path / "main.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "main")], check=True, capture_output=True, text=True, timeout=60).stdout
    assert out.split() == ["200", "7", "200"]
