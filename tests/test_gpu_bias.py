"""GPU test of the FP32 fused arm's mean error against FP64 at padded rank 32: the two
contractions of a half-iteration truncate and their errors have to offset each other.

An MMA step truncates its sums of positive terms by half a unit of 2^-23 on the mean, at
the size the sum has reached.  D = X Y^T: four TF32 steps at 1/4 .. 4/4 of it, then four
BF16 steps at all of it, 6.5 halves; R Y: one step at 1/8, four small ones there, seven at
2/8 .. 8/8, 5 halves.  They offset to 1.5 halves of 2^-23 at most = 1.5 * 2^-24 (below rank
32 D's steps differ by less than that: a step of padding columns truncates nothing).  With
D's small terms first it has 2.75 halves and the difference is 2.25.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [17, 20, 24, 28, 32])
def test_truncations_offset(pkg, k):
    import torch

    n, m = 9001, 801
    g = torch.Generator(device="cuda").manual_seed(k)
    W0 = torch.exp(torch.randn(n, k, device="cuda", generator=g))
    H0 = 0.1 * torch.rand(k, m, device="cuda", generator=g)
    H0[torch.randint(k, (m,), device="cuda", generator=g), torch.arange(m, device="cuda")] = 1.0
    V = torch.poisson(50.0 * (W0 @ H0), generator=g)
    torch.cuda.synchronize()
    rng = np.random.default_rng(k)
    W, H = (rng.random((r, k), np.float32) + np.finfo(np.float32).tiny for r in (n, m))
    V64, W64, H64 = V.double(), torch.from_numpy(W).cuda().double(), torch.from_numpy(H).cuda().double()

    def mean_error(got, want):
        return abs((torch.from_numpy(got).cuda().double() / want - 1).mean().item()) * 2.0 ** 24

    with pkg.NMF(n, m, k) as e:
        e.set_V_device(V.data_ptr(), m)
        e.set_WH(W, H)
        e.update_H()
        H1 = e.H
        e.update_W()
        W1 = e.W
    assert mean_error(H1, H64 * ((V64 / (W64 @ H64.T)).T @ W64) / W64.sum(0)) <= 1.5
    H64 = torch.from_numpy(H1).cuda().double()
    assert mean_error(W1, W64 * ((V64 / (W64 @ H64.T)) @ H64) / H64.sum(0)) <= 1.5
