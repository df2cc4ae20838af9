"""GPU test of the consensus summary with more samples than its kernel has threads (1024):
several slots a thread in the search and the update of a merge, most distances tied, and
a merge after which more rows than the list holds (1024) have lost their nearest slot.

The merges take the lowest pair of slots on ties and the heights are the same FP64
operations in the same order; the sums of the correlation have 1e6 terms: 1e-10.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _linkage(D):
    """Cophenetic distances of average linkage, the lowest pair of slots on ties (rows keep their nearest slot)."""
    m = D.shape[0]
    idx, size, when, into, height = np.arange(m), np.ones(m), np.full(m, m), np.zeros(m, int), []
    left = np.where(idx[None, :] > idx[:, None], D, np.inf)
    near, dist = left.argmin(1), left.min(1)
    for step in range(m - 1):
        a = int(dist.argmin())
        b = int(near[a])
        height.append(dist[a])
        row = (size[a] * D[a] + size[b] * D[b]) / (size[a] + size[b])
        size[a] += size[b]
        size[b] = 0
        when[b], into[b] = step, a
        D[a], D[:, a] = row, row
        alive = size > 0
        left[a] = np.where((idx > a) & alive, row, np.inf)
        left[:, a] = np.where((idx < a) & alive, row, np.inf)
        left[b], left[:, b], dist[b] = np.inf, np.inf, np.inf
        again = np.flatnonzero(alive & ((near == a) | (near == b) | (idx == a)))
        near[again], dist[again] = left[again].argmin(1), left[again].min(1)
        closer = alive & (idx < a) & ((row < dist) | ((row == dist) & (a < near)))
        near[closer], dist[closer] = a, row[closer]
    coph, height = np.zeros((m, m)), np.array(height + [0.0, 0.0])   # (two more for slots that are never absorbed)
    for i in range(m):
        x, y, h = np.full(m, i), idx.copy(), np.zeros(m)
        while (x != y).any():
            fx, apart = when[x] < when[y], x != y
            h = np.where(apart, height[np.minimum(when[x], when[y])], h)
            x, y = np.where(apart & fx, into[x], x), np.where(apart & ~fx, into[y], y)
        coph[i] = h
    return coph


def _planted(rng, m, runs, noise):
    planted = rng.integers(0, 2, m)
    return np.where(rng.random((runs, m)) < noise, 1 - planted, planted)


def _hub(rng, m, runs, k):
    """Every sample agrees with the last one in 30 % of the runs and with no other as often."""
    labels = rng.integers(1, k, (runs, m))
    for x in range(m):
        labels[rng.permutation(runs)[: runs * 3 // 10], x] = 0
    labels[:, -1] = 0
    return labels


@pytest.mark.parametrize("m,k,runs,noise", [(1100, 2, 2, 0.0), (1600, 2, 3, 0.02), (2000, 2, 5, 0.3), (1100, 8, 200, None)])
def test_more_samples_than_threads(pkg, m, k, runs, noise):
    rng = np.random.default_rng(m)
    labels = _hub(rng, m, runs, k) if noise is None else _planted(rng, m, runs, noise)
    C = sum((labels == c).astype(np.float32).T @ (labels == c).astype(np.float32) for c in range(k)).astype(int)
    D = 1.0 - C / runs
    np.fill_diagonal(D, 0.0)
    if noise is None:   # all rows lose their nearest slot at the first merge
        others = C - runs * np.eye(m, dtype=int)
        assert (others[:-1].argmax(1) == m - 1).all() and m - 2 > 1024
    with pkg.Batch(32, m, [k] * runs) as b:
        b.set_V(np.ones((32, m), np.float32))
        for p in range(runs):
            H = np.full((m, k), 0.1, np.float32)
            H[np.arange(m), labels[p]] = 1.0
            b.set_WH(p, np.full((32, k), 0.5, np.float32), H)
        b.run(1, 1, 40)
        assert np.array_equal(b.classification(), labels)
        counts, n, coph = b.consensus(k)
    assert n == runs and np.array_equal(counts, C)
    tree, up = _linkage(D.copy()), np.triu_indices(m, 1)
    x, y = D[up] - D[up].mean(), tree[up] - tree[up].mean()
    xx, yy = x @ x, y @ y
    assert abs(coph - ((x @ y) / np.sqrt(xx * yy) if xx > 0 and yy > 0 else 0.0)) <= 1e-10
