"""GPU test: threads that ask one batch for the summaries of different ranks at the same
time, the first call with its workspaces among them, get what each gets alone (exact)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_summaries_from_several_threads(pkg):
    m, ranks = 120, [2] * 5 + [3] * 9 + [4] * 2 + [5] * 14

    def batch():
        b = pkg.Batch(60, m, ranks)
        b.set_V(np.random.default_rng(3).poisson(4.0, (60, m)).astype(np.float32))
        b.init_random(range(1, len(ranks) + 1))
        b.run(20, 10, 40)
        return b

    with batch() as b:
        alone = {k: b.consensus(k) for k in (2, 3, 4, 5)}
    wrong = []
    with batch() as b:
        def work(k):
            for _ in range(30):
                counts, runs, coph = b.consensus(k)
                if not (np.array_equal(counts, alone[k][0]) and (runs, coph) == alone[k][1:]):
                    wrong.append(k)

        ts = [threading.Thread(target=work, args=(k,)) for k in (2, 3, 4, 5)]
        [t.start() for t in ts]
        [t.join() for t in ts]
    assert wrong == []
