"""GPU test of the plain arm's long sums: the root mean square error of one update
against FP64 where a split of the reduction has more steps than one FP32 chain may.

Tolerance, in units of 2^-24: a rounding to nearest is off by at most one unit,
uniformly spread, so its variance is at most 1/3.  A chain of N positive terms rounds
partial sums that grow evenly: N/3 roundings of the whole sum's size in variance, and P
chains that are added independently average theirs: (N/3)/P, then P/3 for adding them in
turn.  With R steps in chains of 512 and P = R/512, plus three roundings of product,
division and column sum: rms <= sqrt((512/(3 P) + P/3 + 3) / 3); 3 covers it from R = 5000
to 40000 with half as much again for the quotients.  One chain of 10000 is at 19 and of
5000 at 13 by the same rule.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RMS = 3.0 * 2.0 ** -24


@pytest.mark.parametrize("n,m,k", [(38000, 20000, 129), (39000, 5000, 256), (60000, 300, 130)])
def test_long_reductions_against_fp64(pkg, n, m, k):
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    V = torch.poisson(torch.full((n, m), 6.0, device="cuda"), generator=g)
    torch.cuda.synchronize()
    rng = np.random.default_rng(n)
    W, H = (rng.random((r, k), np.float32) + np.float32(0.05) for r in (n, m))
    Wd, Hd = (torch.from_numpy(x).cuda().double() for x in (W, H))
    rows = 4000   # rows of V a step of the reference

    def rms(got, want):
        return (torch.from_numpy(got).cuda().double() / want - 1).square().mean().sqrt().item()

    with pkg.NMF(n, m, k, arm="plain") as e:
        e.set_V_device(V.data_ptr(), m)
        e.set_WH(W, H)
        e.update_H()
        H1 = e.H
        aux = torch.zeros_like(Hd)
        for i in range(0, n, rows):
            w = Wd[i:i + rows]
            aux += (V[i:i + rows].double() / (w @ Hd.T)).T @ w
        assert rms(H1, Hd * aux / Wd.sum(0)) <= RMS
        e.update_W()
        Hd = torch.from_numpy(H1).cuda().double()
        want = torch.cat([Wd[i:i + rows] * ((V[i:i + rows].double() / (Wd[i:i + rows] @ Hd.T)) @ Hd)
                          for i in range(0, n, rows)]) / Hd.sum(0)
        assert rms(e.W, want) <= RMS


@pytest.mark.parametrize("n,m,k", [(1000, 97, 65), (8000, 1000, 100), (16000, 130, 70)])
def test_many_partials_against_fp64(pkg, n, m, k):
    """update_H from 63 or 64 splits of a few hundred rows at most: by the rule above their chains
    cost (N/3)/64 < 2, and adding them in eights (7 roundings in a tree of 3, then P/8 in turn)
    (P/8)/3 + 1 with product, division and column sum 3: rms <= sqrt((2 + 3.7 + 3) / 3) = 1.7,
    one after another 64/3 -> 2.9."""
    rng = np.random.default_rng(k)
    V = rng.poisson(6.0, (n, m)).astype(np.float32)
    W, H = (rng.random((r, k), np.float32) + np.float32(0.05) for r in (n, m))
    with pkg.NMF(n, m, k, arm="plain") as e:
        e.set_V(V)
        e.set_WH(W, H)
        e.update_H()
        got = e.H
    Wd, Hd = W.astype(np.float64), H.astype(np.float64)
    want = Hd * ((V / (Wd @ Hd.T)).T @ Wd) / Wd.sum(0)
    assert np.sqrt(np.mean((got / want - 1) ** 2)) <= 1.7 * 2.0 ** -24
