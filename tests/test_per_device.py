"""Streams and events that a thread keeps are one set per device: the holder
behind them (csrc/ct_per_device.cuh, plain C++) compiled and run on the CPU,
with a device number in the place of cudaGetDevice's."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cudatree_b200" / "csrc"
MAIN = r"""
#include "ct_per_device.cuh"
#include <cstdio>
#include <thread>
static int made = 0, gone = 0;
struct Set {
  int id;
  Set() : id(made++) {}
  ~Set() { ++gone; }
};
static Set& mine(int device) {
  static thread_local ct::PerDevice<Set> all;
  return all.on(device);
}
int main() {
  Set* a = &mine(0);
  Set* b = &mine(1);
  for (int d = 2; d < 64; ++d) mine(d);
  const bool kept = a == &mine(0) && b == &mine(1) && a != b && made == 64;
  bool other = false;
  std::thread t([&] { other = &mine(0) != a && &mine(1) != b; });
  t.join();
  std::printf("%d %d %d %d\n", kept, other, made, gone);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_one_set_per_thread_and_device(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-pthread", f"-I{CSRC}", "main.cpp", "-o", "main"], cwd=tmp_path, check=True)
    out = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True, check=True).stdout
    # kept for each device, another thread has its own, which end with it
    assert out.split() == ["1", "1", "66", "2"]


def test_fit_keeps_its_capture_streams_per_device():
    """Both of the fit's per-thread stream sets are looked up by the current device."""
    src = (CSRC / "ct_fit.cu").read_text()
    for name in ("cudaStream_t capture_stream()", "const ForkStreams* fork_streams()"):
        body = src[src.index(name):]
        body = body[:body.index("\n}\n")]
        assert "thread_local PerDevice<" in body and "cudaGetDevice(&dev)" in body and "all.on(dev)" in body
