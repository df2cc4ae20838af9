"""GPU test of nmfb_set_sm_limit's purpose: a large context limited to part of the
device leaves SMs on which another context's kernels run while its own do.

Rates of the same small context beside the large one, limited and not. With 37 SMs
free for the whole of every large kernel instead of the gaps between them the small
context gets several times as much; half as much again is asked for.
"""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_limit_leaves_room_for_others(pkg):
    import torch

    n, m, k = 60000, 2000, 20
    rng = np.random.default_rng(1)
    V = torch.poisson(torch.full((n, m), 5.0, device="cuda"))
    small_V = rng.poisson(5.0, (5000, 38)).astype(np.float32)
    torch.cuda.synchronize()

    def factors(rows, cols, rank):
        return [rng.random((r, rank), np.float32) + np.float32(0.05) for r in (rows, cols)]

    def small_runs(limit):
        with pkg.NMF(n, m, k) as large, pkg.NMF(5000, 38, 3) as small:
            large.set_sm_limit(limit)
            large.set_V_device(V.data_ptr(), m)
            large.set_WH(*factors(n, m, k))
            small.set_V(small_V)
            small.set_WH(*factors(5000, 38, 3))
            large.run(20, 10, 10 ** 6)
            small.run(20, 10, 10 ** 6)
            runs = [0, 0]
            end = time.perf_counter() + 0.5

            def work(i, e):
                while time.perf_counter() < end:
                    e.run(20, 10, 10 ** 6)
                    runs[i] += 1

            ts = [threading.Thread(target=work, args=a) for a in ((0, large), (1, small))]
            [t.start() for t in ts]
            [t.join() for t in ts]
            assert runs[0] > 0
            return runs[1]

    assert small_runs(111) >= 1.5 * small_runs(0)
