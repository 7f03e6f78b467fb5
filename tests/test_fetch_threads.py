"""Host threads of the tree read-back (CPU)."""
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "cudatree_b200" / "csrc"


def test_copying_threads_are_on_the_callers_device():
    """A thread starts on device 0: its first runtime call would make a context
    there, whatever device the caller's fit is on."""
    src = (CSRC / "ct_fit.cu").read_text()
    body = src[src.index("auto copy = [&](uint32_t w) {"):]
    body = body[:body.index("\n    };")]
    assert 0 < body.index("cudaSetDevice(dev)") < body.index("cudaEventSynchronize")
