"""GPU test of the fetch of a batch's factors through bounded staging: the values over
several chunks (exact), and the page-locked memory that a fetch leaves in the pool."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned():
    with open("/proc/self/status") as f:   # page-locked buffers count as shared memory
        return next(int(line.split()[1]) for line in f if line.startswith("RssShmem")) * 1024


@pytest.mark.parametrize("n,k", [(1000000, 20), (262144, 8), (262145, 6), (600001, 5), (7, 3)])
def test_factors_come_back_whole(pkg, n, k):
    m = 40
    rng = np.random.default_rng(k)
    W, H = rng.random((n, k), np.float32), rng.random((m, k), np.float32)
    with pkg.Batch(n, m, [2, k]) as b:
        b.set_WH(1, W, H)
        pkg.load_library().nmfb_release_cached(0)
        before = _pinned()
        assert np.array_equal(b.W(1), W) and np.array_equal(b.H(1), H)
        # two buffers of 8 MB and one for H's 4 KB, and 4 MB for whatever else the process does
        assert _pinned() - before <= 20 * 1024 * 1024
