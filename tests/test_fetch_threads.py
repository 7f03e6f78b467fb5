"""Host threads of the tree read-back (CPU)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cudatree_b200" / "csrc"


def test_copying_threads_are_on_the_callers_device():
    """A thread starts on device 0: its first runtime call would make a context
    there, whatever device the caller's fit is on."""
    src = (CSRC / "ct_fit.cu").read_text()
    body = src[src.index("auto copy = [&](uint32_t w) {"):]
    body = body[:body.index("\n    };")]
    assert 0 < body.index("cudaSetDevice(dev)") < body.index("cudaEventSynchronize")


MAIN = r"""
#include "ct_parts.h"
#include <cstdio>
#include <stdexcept>
#include <system_error>
#include <utility>
static int left = 0;  // threads that can still be started
struct Few : std::thread {
  template <typename F>
  Few(F& f, uint32_t& i) : std::thread(take(f), i) {}
  template <typename F>
  static F& take(F& f) {
    if (left-- <= 0) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
    return f;
  }
};
int main() {
  for (int can : {0, 1, 3, 16}) {
    left = can;
    int runs[8] = {};
    ct::run_parts<Few>(8, [&](uint32_t i) { ++runs[i]; });
    for (int r : runs) std::printf("%d", r);
    std::printf(" ");
  }
  for (uint32_t bad : {0u, 2u, 7u}) {  // a part that throws: the others have ended when the caller sees it
    left = 3;
    int runs[8] = {};
    try {
      ct::run_parts<Few>(8, [&](uint32_t i) {
        if (i == bad) throw std::runtime_error("part");
        ++runs[i];
      });
      std::printf("none ");
    } catch (const std::runtime_error& e) {
      int sum = 0;
      for (int r : runs) sum += r;
      std::printf("%s%d ", e.what(), sum);
    }
  }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_every_part_runs_when_threads_are_short(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-pthread", f"-I{CSRC}", "main.cpp", "-o", "main"], cwd=tmp_path, check=True)
    out = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True, check=True).stdout
    assert out.split() == ["11111111"] * 4 + ["part7"] * 3
