"""GPU tests of the FP64 objectives of matrices with few columns: the edges of the
tiles that 1 to 4, 5 to 16, 17 to 32 and more columns get, and that a narrow matrix
does not take several times as long as a wide one of as many elements.

Both sides sum the same FP64 terms in other orders; over the at most 1.2e5 elements
here they agree to 1.2e5 * 2^-53 of the sum of the terms' magnitudes, below 1e-9.
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,k", [(2, 2, 2), (1023, 3, 2), (1025, 4, 4), (255, 5, 5), (257, 16, 16), (600, 17, 17),
                                   (127, 32, 31), (129, 33, 33), (30000, 4, 3)])
def test_objectives_of_narrow_matrices(pkg, oracle, n, m, k):
    rng = np.random.default_rng(n * 1000 + m)
    V = rng.poisson(3.0, (n, m)).astype(np.float32)
    W = rng.random((n, k), np.float32) + np.float32(0.01)
    H = rng.random((m, k), np.float32) + np.float32(0.01)
    WH = W.astype(np.float64) @ H.T.astype(np.float64)
    with pkg.NMF(n, m, k) as e:
        e.set_V(V)
        e.set_WH(W, H)
        vv, dd = e.dot_product_VWH()
        kl = e.kl_divergence()
    V64 = V.astype(np.float64)
    assert abs(vv - (V64 ** 2).sum()) <= 1e-9 * (V64 ** 2).sum()
    assert abs(dd - ((V64 - WH) ** 2).sum()) <= 1e-9 * ((V64 - WH) ** 2).sum()
    want = oracle.kl_divergence(V, W, H)
    assert abs(kl - want) <= 1e-9 * (np.abs(V64 - WH).sum() + abs(want))


def test_narrow_takes_no_longer(pkg):
    """Two million elements either way; twice the traffic in the narrow one's padded rows and
    a wider W leave room for a factor of 3 (64-column tiles took 7 times as long)."""
    def seconds(n, m):
        rng = np.random.default_rng(m)
        with pkg.NMF(n, m, 2) as e:
            e.set_V(rng.poisson(3.0, (n, m)).astype(np.float32))
            e.set_WH(*(rng.random((r, 2), np.float32) + np.float32(0.01) for r in (n, m)))
            times = []
            for _ in range(15):
                t = time.perf_counter()
                e.kl_divergence()
                times.append(time.perf_counter() - t)
        return sorted(times)[7]

    assert seconds(1000000, 2) <= 3.0 * seconds(2000, 1000)
