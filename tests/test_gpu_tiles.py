"""GPU tests of the fused kernels' tile lists: runs of tiles that cross row
blocks, start inside one, cover many one-tile row blocks or fill single CTAs,
with ragged last tiles; every update against FP64 of the same inputs.

Tolerances: the quotient's denominator and both contractions carry at most
2^-20 of relative error per product in the FP32 arm (TF32 main terms, small
terms to 2^-9) and 2^-16 in split BF16, and the sums of positive terms do not
amplify it: 4 * 2^-20 and 4 * 2^-16 bound an update's entries.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"fused": 4 * 2.0 ** -20, "bf16x3": 4 * 2.0 ** -16}


def _updates(V, W, H):
    V, W, H = (x.astype(np.float64) for x in (V, W, H))
    H1 = H * ((V / (W @ H.T)).T @ W) / W.sum(0)
    return H1


@pytest.mark.parametrize("arm", ["fused", "bf16x3"])
@pytest.mark.parametrize("n,m,k,sms", [
    (129, 65, 3, 0),        # two row blocks, ragged tiles on both sides
    (129, 65, 30, 0),       # (the FP32 arm's tensor-core kernels)
    (2000, 33, 5, 0),       # one-tile row blocks (W side), one CTA each
    (2000, 33, 27, 0),      # (the FP32 arm's tensor-core kernels from here on)
    (3000, 40, 16, 5),      # one-tile row blocks, several to a CTA
    (5000, 130, 20, 7),     # three-tile row blocks crossed by runs of every phase
    (9000, 70, 33, 3),      # rank 64 instantiation: 64-column tiles, a single X buffer
    (700, 9000, 17, 2),     # long reductions: partials every 128 tiles
    (8320, 300, 2, 1),      # one CTA does everything
    (16400, 129, 64, 148),  # partial sums that end on a multiple of 128 tiles
])
def test_update_against_fp64(pkg, arm, n, m, k, sms):
    rng = np.random.default_rng(n + m + k)
    V = rng.poisson(5.0, (n, m)).astype(np.float32)
    W = rng.random((n, k), np.float32) + np.float32(0.05)
    H = rng.random((m, k), np.float32) + np.float32(0.05)
    with pkg.NMF(n, m, k, arm=arm) as e:
        e.set_sm_limit(sms)
        e.set_V(V)
        for _ in range(3):      # the same answer every time
            e.set_WH(W, H)
            e.update_H()
            H1 = e.H
            want = _updates(V, W, H)
            assert np.abs(H1 / want - 1).max() <= TOL[arm]
            e.update_W()
            want = _updates(V.T, H1, W)
            assert np.abs(e.W / want - 1).max() <= TOL[arm]


@pytest.mark.parametrize("arm,k", [("bf16x3", 40), ("bf16x3", 32), ("split_bf16", 64), ("fused", 50), ("fused", 20), ("bf16", 64)])
def test_long_runs_end_alike(pkg, arm, k):
    """Many tiles per CTA with loads that land out of order (V larger than L2): the R
    teams' uses of a V stage must not run into one another, run after run."""
    import torch

    n, m = 30001, 3001
    g = torch.Generator(device="cuda").manual_seed(k)
    V = torch.poisson(torch.full((n, m), 6.0, device="cuda"), generator=g)
    torch.cuda.synchronize()
    rng = np.random.default_rng(k)
    W, H = (rng.random((r, k), np.float32) + np.float32(0.05) for r in (n, m))
    with pkg.NMF(n, m, k, arm=arm) as e:
        e.set_V_device(V.data_ptr(), m)
        first = None
        for _ in range(8):
            e.set_WH(W, H)
            assert e.run(40, 10, 10 ** 6) == (40, False)
            got = e.W, e.H
            first = first or got
            assert all(np.array_equal(a, b) for a, b in zip(got, first))
