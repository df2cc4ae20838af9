"""GPU tests of the FP32 SIMT kernels at tile edges: the plain arm's 128 x 64
tiles with 16 reduction steps (rows, columns, ranks and split reductions that
end inside one) and the no-allocation update at every rank class and row group.
One update against FP64 of the same inputs: sums of positive FP32 terms in
chains of at most 512 with a quotient of 2 ulp, 3e-5 relative at worst
(512 * 2^-24).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 3e-5


def _inputs(n, m, k):
    rng = np.random.default_rng(n + 7 * m + 13 * k)
    V = rng.poisson(4.0, (n, m)).astype(np.float32)
    return V, rng.random((n, k), np.float32) + np.float32(0.05), rng.random((m, k), np.float32) + np.float32(0.05)


def _update(V, W, H):
    V, W, H = (x.astype(np.float64) for x in (V, W, H))
    return H * ((V / (W @ H.T)).T @ W) / W.sum(0)


@pytest.mark.parametrize("n,m,k", [(2, 2, 2), (127, 65, 15), (128, 64, 16), (129, 63, 17), (1000, 97, 65), (513, 130, 97),
                                   (4097, 260, 129), (300, 2000, 256)])
def test_plain_update_against_fp64(pkg, n, m, k):
    V, W, H = _inputs(n, m, k)
    with pkg.NMF(n, m, k, arm="plain") as e:
        e.set_V(V)
        e.set_WH(W, H)
        e.update_H()
        H1 = e.H
        assert np.abs(H1 / _update(V, W, H) - 1).max() <= TOL
        e.update_W()
        assert np.abs(e.W / _update(V.T, H1, W) - 1).max() <= TOL


@pytest.mark.parametrize("n,m,k", [(1, 1, 1), (5, 129, 3), (31, 128, 4), (33, 127, 7), (700, 300, 13), (64, 1025, 20),
                                   (1201, 130, 30), (9000, 40, 41), (500, 257, 53), (2049, 65, 64)])
def test_noalloc_against_fp64(pkg, n, m, k):
    import torch

    V, W, H = _inputs(n, m, k)
    # rows on odd pitches: nothing about the caller's buffers is aligned but the values
    dV, dW, dH = (torch.zeros(x.shape[0], x.shape[1] + p, device="cuda") for x, p in ((V, 3), (W, 1), (H, 2)))
    dV[:, :m], dW[:, :k], dH[:, :k] = (torch.from_numpy(x).cuda() for x in (V, W, H))
    torch.cuda.synchronize()
    pkg.update_H_noalloc(dV.data_ptr(), m + 3, dW.data_ptr(), k + 1, dH.data_ptr(), k + 2, n, m, k,
                         torch.cuda.current_stream().cuda_stream)
    got = dH.cpu().numpy()
    assert np.abs(got[:, :k] / _update(V, W, H) - 1).max() <= TOL
    assert (got[:, k:] == 0).all()
