"""GPU test of the consensus summary against a direct average linkage: many tied
distances (few runs), no ties, two samples, one cluster, more samples than a
merge step scans at a time.  The merges take the lowest pair of slots on
ties and the heights are the same FP64 operations in the same order, so the
correlation agrees to the rounding of its sums (at most m^2 terms: 1e-10).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(labels):
    runs, m = labels.shape
    C = (labels[:, :, None] == labels[:, None, :]).sum(0)
    D = 1.0 - C / runs
    np.fill_diagonal(D, 0.0)
    full, size, members = D.copy(), np.ones(m), [[i] for i in range(m)]
    left = D.copy()
    left[np.tril_indices(m)] = np.inf
    coph, idx = np.zeros((m, m)), np.arange(m)
    for _ in range(m - 1):
        a, b = divmod(int(np.argmin(left)), m)      # the first minimum: the lowest pair
        coph[np.ix_(members[a], members[b])] = left[a, b]
        coph[np.ix_(members[b], members[a])] = left[a, b]
        row = (size[a] * full[a] + size[b] * full[b]) / (size[a] + size[b])
        members[a] += members[b]
        size[a] += size[b]
        size[b] = 0
        full[a], full[:, a] = row, row
        left[a] = np.where((idx > a) & (size > 0), row, np.inf)
        left[:, a] = np.where((idx < a) & (size > 0), row, np.inf)
        left[b], left[:, b] = np.inf, np.inf
    up = np.triu_indices(m, 1)
    x, y = D[up] - D[up].mean(), coph[up] - coph[up].mean()
    xx, yy = x @ x, y @ y
    return C, (x @ y) / np.sqrt(xx * yy) if xx > 0 and yy > 0 else 0.0


@pytest.mark.parametrize("m,k,runs,noise", [(2, 2, 3, 0.5), (3, 2, 4, 0.5), (33, 3, 2, 0.3), (64, 5, 1, 0.0),
                                            (150, 4, 37, 0.4), (257, 8, 20, 1.0), (300, 2, 5, 0.05)])
def test_cophenetic_against_direct_linkage(pkg, m, k, runs, noise):
    rng = np.random.default_rng(m)
    planted = rng.integers(0, k, m)
    moved = rng.random((runs, m)) < noise
    labels = np.where(moved, rng.integers(0, k, (runs, m)), planted[None, :])
    with pkg.Batch(32, m, [k] * runs) as b:
        b.set_V(np.ones((32, m), np.float32))
        for p in range(runs):                       # H keeps the order of its columns on a constant matrix
            H = np.full((m, k), 0.1, np.float32)
            H[np.arange(m), labels[p]] = 1.0
            b.set_WH(p, np.full((32, k), 0.5, np.float32), H)
        b.run(1, 1, 40)
        assert np.array_equal(b.classification(), labels)
        counts, n, coph = b.consensus(k)
        again = b.consensus(k)[2]                   # the workspace is used again
    C, want = _reference(labels)
    assert n == runs and np.array_equal(counts, C)
    assert abs(coph - want) <= 1e-10 and coph == again
