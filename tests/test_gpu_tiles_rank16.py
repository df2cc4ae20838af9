"""GPU tests of the FP32 fused kernels at padded rank 16 (their own small terms, buffers
and V ring) on shapes that the small-matrix kernels do not take: ragged tiles on both
sides of two row blocks, one-tile row blocks with a CTA each, single rows over a block.
The launches show which kernels ran: three for a single update of the fused ones.

Tolerance as for the other ranks: 4 * 2^-20 of an entry (2^-20 per product).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _update(V, W, H):
    V, W, H = (x.astype(np.float64) for x in (V, W, H))
    return H * ((V / (W @ H.T)).T @ W) / W.sum(0)


@pytest.mark.parametrize("n,m,k", [(300, 193, 16), (193, 300, 11), (129, 257, 9), (60, 2000, 5), (64, 1025, 4), (2000, 520, 2)])
def test_update_against_fp64(pkg, n, m, k):
    rng = np.random.default_rng(n + m + k)
    V = rng.poisson(5.0, (n, m)).astype(np.float32)
    W = rng.random((n, k), np.float32) + np.float32(0.05)
    H = rng.random((m, k), np.float32) + np.float32(0.05)
    with pkg.NMF(n, m, k) as e:
        e.set_V(V)
        for _ in range(3):
            e.set_WH(W, H)
            launches = e.launch_count()
            e.update_H()
            H1 = e.H
            assert e.launch_count() - launches == 3
            assert np.abs(H1 / _update(V, W, H) - 1).max() <= 4 * 2.0 ** -20
            e.update_W()
            assert e.launch_count() - launches == 6
            assert np.abs(e.W / _update(V.T, H1, W) - 1).max() <= 4 * 2.0 ** -20
