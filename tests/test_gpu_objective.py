"""GPU tests of the FP64 objectives over tile edges and rank chunks: 64 x 64
tiles of V, 32 columns of the factors at a time, and the kernels that form only
the dots or only the divergence.  Both sides sum the same FP64 terms in other
orders; over the at most 1e5 elements here the sums agree to 1e5 * 2^-53 of
the sum of the terms' magnitudes, below 1e-9 of the results.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,k,arm", [(2, 2, 2, "fused"), (63, 65, 31, "fused"), (64, 64, 32, "fused"),
                                       (65, 63, 33, "fused"), (257, 190, 64, "fused"), (300, 129, 100, "plain")])
def test_objectives_at_tile_edges(pkg, oracle, n, m, k, arm):
    rng = np.random.default_rng(n * 1000 + m)
    V = rng.poisson(3.0, (n, m)).astype(np.float32)      # exact zeros among them
    W = rng.random((n, k), np.float32) + np.float32(0.01)
    H = rng.random((m, k), np.float32) + np.float32(0.01)
    WH = W.astype(np.float64) @ H.T.astype(np.float64)
    with pkg.NMF(n, m, k, arm=arm) as e:
        e.set_V(V)
        e.set_WH(W, H)
        vv, dd = e.dot_product_VWH()
        kl = e.kl_divergence()
    V64 = V.astype(np.float64)
    assert abs(vv - (V64 ** 2).sum()) <= 1e-9 * (V64 ** 2).sum()
    assert abs(dd - ((V64 - WH) ** 2).sum()) <= 1e-9 * ((V64 - WH) ** 2).sum()
    want = oracle.kl_divergence(V, W, H)
    assert abs(kl - want) <= 1e-9 * (np.abs(V64 - WH).sum() + abs(want))
