"""GPU tests of the two-launch half-iterations of small matrices: ranks at every
padded width, fewer rows than SMs, ragged slabs, one and several thread groups,
a limited SM count, and the sizes next to the rule's limits.

Tolerance: FP32 sums of positive terms, in chains of at most 512 per thread, then
groups and CTAs, and a quotient of 2 ulp: 3e-5 relative per update at worst
(512 * 2^-24), and far less on average.
"""
import threading

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


SHAPES = [(2, 2, 2, 0), (147, 33, 3, 0), (149, 2, 2, 0), (5, 512, 4, 0), (1000, 256, 5, 0), (3001, 170, 9, 0),
          (17900, 128, 16, 0), (700, 102, 20, 0), (19500, 85, 24, 0), (2500, 40, 22, 37), (300, 24, 24, 1)]


@pytest.mark.parametrize("n,m,k,sms", SHAPES)
def test_updates_against_fp64(pkg, n, m, k, sms):
    V, W, H = _inputs(n, m, k)
    with pkg.NMF(n, m, k) as e:
        e.set_sm_limit(sms)
        e.set_V(V)
        e.set_WH(W, H)
        l0 = e.launch_count()
        e.update_H()
        H1 = e.H
        e.update_W()
        assert e.launch_count() - l0 == 3          # the path under test: two launches and one
        assert np.abs(H1 / _update(V, W, H) - 1).max() <= TOL
        assert np.abs(e.W / _update(V.T, H1, W) - 1).max() <= TOL


@pytest.mark.parametrize("n,m,k,sms", [(147, 33, 3, 0), (3001, 170, 9, 0), (19500, 85, 24, 0), (2500, 40, 22, 37)])
def test_run_is_its_steps(pkg, n, m, k, sms):
    """A run (graph blocks, the next update_H's sums formed by update_W's launch) gives
    the single steps' factors bit for bit, with and without profiling, and stops alike."""
    V, W, H = _inputs(n, m, k)
    with pkg.NMF(n, m, k) as e:
        e.set_sm_limit(sms)
        e.set_V(V)
        e.set_WH(W, H)
        for i in range(23):
            e.update_H()
            e.update_W()
            if (i + 1) % 10 == 0:
                e.adjust()
        Ws, Hs = e.W, e.H
        for profile in (False, True, False):
            e.profile(profile)
            e.set_WH(W, H)
            assert e.run(23, 10, 10 ** 6) == (23, False)
            assert np.array_equal(e.W, Ws) and np.array_equal(e.H, Hs)
        e.set_WH(W, H)
        it, conv = e.run(10000, 10, 1)
        assert conv and it % 10 == 0 and it < 10000
        Wc = e.W
        e.set_WH(W, H)
        e.run(it, 10, 10 ** 6)
        assert np.array_equal(e.W, Wc)             # nothing ran after the stop


def test_many_contexts_at_once(pkg):
    """Results alone and among eleven other contexts of other sizes are the same."""
    shapes = [(1000 + 517 * i, 20 + 7 * i, 2 + i % 11) for i in range(12)]
    es, alone = [], []
    for n, m, k in shapes:
        V, W, H = _inputs(n, m, k)
        e = pkg.NMF(n, m, k)
        e.set_V(V)
        e.set_WH(W, H)
        e.run(60, 10, 10 ** 6)
        alone.append((e.W, e.H))
        es.append((e, W, H))
    got = [None] * 12

    def work(i):
        e, W, H = es[i]
        for _ in range(5):
            e.set_WH(W, H)
            e.run(60, 10, 10 ** 6)
        got[i] = (e.W, e.H)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(12)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    for (W, H), (Wa, Ha) in zip(got, alone):
        assert np.array_equal(W, Wa) and np.array_equal(H, Ha)
    [e.close() for e, _, _ in es]
