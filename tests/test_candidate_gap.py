"""The scan's candidate test (ct_common.cuh, is_candidate_sorted) decides most
neighbours by their float gap: every decision must be the double test's
(x + 1e-5 < x_next, the reference's dfs_module.cu:400)."""
import numpy as np


def _fast(x, xn):
    exact = x.astype(np.float64) + 0.00001 < xn.astype(np.float64)
    with np.errstate(over="ignore", invalid="ignore"):
        gap = xn - x
    return np.where(~(xn > x), False,
                    np.where(gap > np.float32(1.00001e-5), True, np.where(gap < np.float32(0.99999e-5), False, exact)))


def test_gap_decides_as_the_double_test():
    rng = np.random.default_rng(11)
    base = np.concatenate([rng.normal(size=4000), rng.normal(size=4000) * 1e-5, rng.uniform(-300, 300, 4000),
                           rng.normal(size=2000) * 1e6, rng.normal(size=500) * 1e30, rng.normal(size=500) * 1e-30,
                           [0.0, -0.0, np.inf, -np.inf, 127.99999, 128.0, -128.0, 3.4e38, -3.4e38, 1e-45]]).astype(np.float32)
    pairs = [(base, np.full_like(base, np.inf)), (np.full_like(base, -np.inf), base), (base, base)]
    for steps in (1, 2, 3, 7, 100):
        up = base.copy()
        for _ in range(steps):
            up = np.nextafter(up, np.float32(np.inf))
        pairs.append((base, up))
    for gap in (9.9998e-6, 9.9999e-6, 1e-5, 1.00001e-5, 1.00002e-5, 1e-4, 1.0):
        centre = (base.astype(np.float64) + gap).astype(np.float32)
        for k in range(-4, 5):
            near = centre.copy()
            for _ in range(abs(k)):
                near = np.nextafter(near, np.float32(np.inf if k > 0 else -np.inf))
            pairs.append((base, near))
    for x, xn in pairs:
        ok = xn >= x  # sorted neighbours
        exact = x.astype(np.float64) + 0.00001 < xn.astype(np.float64)
        np.testing.assert_array_equal(_fast(x[ok], xn[ok]), (exact & (xn > x))[ok])
