"""The one-launch presort (a CTA per feature) at its size classes' edges
against a stable argsort, and the one-launch feature flags through fits."""
import numpy as np
import pytest

from . import gpu_utils as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,index_bytes", [(1, 2), (31, 2), (33, 4), (255, 2), (257, 2), (2047, 2), (2048, 4), (2049, 2),
                                           (8191, 2), (8192, 2), (8193, 4), (10000, 2), (16384, 2), (16385, 2)])
def test_presort_is_a_stable_argsort(cuda_device, n, index_bytes):
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 9)).astype(np.float32)
    x[:, 1] = np.round(x[:, 1], 1)
    x[:, 2] = rng.integers(0, 2, n)
    x[:, 3] = -7.25
    x[:, 4] = np.where(rng.random(n) < 0.5, -0.0, 0.0)
    x[:, 5] *= 1e30
    x[::5, 5] = np.inf
    x[1::7, 5] = -np.inf
    x[:, 6] = rng.integers(0, 70000, n)
    x[:, 7] = np.arange(n, 0, -1)
    gp = G.GpuProblem(x, np.zeros(n, np.int64), 1, 1, index_bytes=index_bytes)
    np.testing.assert_array_equal(gp.presort_np(), np.argsort(x.T + 0.0, axis=1, kind="stable"))
