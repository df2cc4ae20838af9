"""The work that users of this framework have it do, as cases to be timed.

Kinds of case and what they stand for:

run        the solver's loop on a resident matrix (``NMF.run``): test blocks of
           ten iterations with the EPS adjust, classification and stop rule, on
           any update arm and rank; the factors go on from the previous pass
step       a program that drives the update entry points itself and watches the
           objective after every iteration (``update_H``, ``update_W``,
           ``kl_divergence``)
noalloc    ``update_H_noalloc`` on buffers of a host framework
sweep      rank selection: many solves of one matrix, one per rank and restart,
           in one launch (``Batch.run``); every restart's H (the memberships) and
           each rank's first restart's W
consensus  the summary of one rank's restarts: co-clustering counts and the
           cophenetic correlation
solve      ``nmf_gpu``: host matrix in; factors and distance out

Sizes are those of the repository's configurations and tests: 5000 x 38 at
rank 3 (an expression matrix), 20000 x 1000 at rank 16, 60000 x 5000 at rank 32
and 64 (counts), a sweep of ranks 2 to 10 over 5000 x 200, requests of 1000 to
50000 rows and 20 to 2000 columns at ranks 2 to 20, ranks above 64 on the plain
arm; and odd ones between them.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

nmf = importlib.import_module("bionmf-gpu_b200")

FLT_MIN = float(np.finfo(np.float32).tiny)
J = 10   # iterations between convergence tests (the command line's default)


def listed():
    return [
        # the reference's own example: a small expression matrix, a rank of few classes
        {"name": "run 5000x38 k3", "kind": "run", "arm": "fused", "n": 5000, "m": 38, "k": 3, "iters": 20},
        # a mid-sized request of a serving mix: ragged in every dimension
        {"name": "run 9973x127 k7", "kind": "run", "arm": "fused", "n": 9973, "m": 127, "k": 7, "iters": 20},
        # a large expression matrix
        {"name": "run 20000x1000 k16", "kind": "run", "arm": "fused", "n": 20000, "m": 1000, "k": 16, "iters": 20},
        # the headline benchmark: counts, one test block
        {"name": "run 60000x5000 k32", "kind": "run", "arm": "fused", "n": 60000, "m": 5000, "k": 32, "iters": 10},
        # an odd rank of the widest fused instantiation
        {"name": "run 40009x3001 k50", "kind": "run", "arm": "fused", "n": 40009, "m": 3001, "k": 50, "iters": 10},
        # the split-BF16 arm, chosen for its speed at FP32-class accuracy
        {"name": "run bf16x3 50000x2000 k20", "kind": "run", "arm": "bf16x3", "n": 50000, "m": 2000, "k": 20, "iters": 10},
        # a rank that only the unfused FP32 arm takes
        {"name": "run plain 8000x1000 k100", "kind": "run", "arm": "plain", "n": 8000, "m": 1000, "k": 100, "iters": 10},
        # single update calls with the objective watched
        {"name": "step 12007x1501 k20", "kind": "step", "arm": "fused", "n": 12007, "m": 1501, "k": 20},
        # one update inside a program that owns the device memory
        {"name": "noalloc 20000x1000 k20", "kind": "noalloc", "n": 20000, "m": 1000, "k": 20},
        # rank selection: ranks 2 to 10, twenty restarts of each
        {"name": "sweep 5000x200 k2-10 x20", "kind": "sweep", "n": 5000, "m": 200, "k": 2, "kmax": 10, "restarts": 20, "iters": 40},
        # the summary of 50 restarts of 200 samples
        {"name": "consensus 200 x50", "kind": "consensus", "m": 200, "k": 5, "restarts": 50},
        # one whole call from host data
        {"name": "solve 10000x250 k8", "kind": "solve", "n": 10000, "m": 250, "k": 8, "iters": 30},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "run", "plain", "step", "noalloc", "sweep", "consensus", "solve"])
    if kind == "run":
        while True:
            n, m, k = _log_int(rng, 1000, 60000), _log_int(rng, 20, 5000), rng.randint(2, 64)
            if k <= m and n * m <= 2.5e8:
                break
        arm = rng.choice(["fused", "fused", "fused", "bf16x3"])
        return {"kind": kind, "arm": arm, "n": n, "m": m, "k": k, "iters": 20 if n * m < 4e7 else 10}
    if kind == "plain":
        return {"kind": "run", "arm": "plain", "n": _log_int(rng, 1000, 12000), "m": _log_int(rng, 130, 1200), "k": rng.randint(65, 128), "iters": 10}
    if kind == "step":
        return {"kind": kind, "arm": "fused", "n": _log_int(rng, 1000, 30000), "m": _log_int(rng, 65, 2000), "k": rng.randint(2, 64)}
    if kind == "noalloc":
        return {"kind": kind, "n": _log_int(rng, 500, 50000), "m": _log_int(rng, 65, 2000), "k": rng.randint(2, 64)}
    if kind == "sweep":
        k = rng.randint(2, 8)
        return {"kind": kind, "n": _log_int(rng, 500, 5000), "m": rng.randint(30, 250), "k": k, "kmax": k + rng.randint(0, 8), "restarts": rng.randint(2, 20), "iters": 40}
    if kind == "consensus":
        return {"kind": kind, "m": rng.randint(30, 400), "k": rng.randint(2, 10), "restarts": rng.randint(5, 50)}
    return {"kind": kind, "n": _log_int(rng, 1000, 20000), "m": _log_int(rng, 20, 500), "k": rng.randint(2, 20), "iters": 30}


# ---- inputs -----------------------------------------------------------------

def _matrix(c, seed):
    """V (n x m, FP32, on the GPU): planted counts, Poisson(50 W0 H0) with lognormal W0 and one dominant class per sample."""
    n, m, k = c["n"], c["m"], min(c["k"], 32)
    g = torch.Generator(device="cuda").manual_seed(seed)
    W0 = torch.exp(torch.randn(n, k, device="cuda", generator=g))
    H0 = 0.1 * torch.rand(k, m, device="cuda", generator=g)
    H0[torch.randint(k, (m,), device="cuda", generator=g), torch.arange(m, device="cuda")] = 1.0
    return torch.poisson(50.0 * (W0 @ H0), generator=g)


def _factors(c, seed, k=None):
    """Initial W (n x k) and H (m x k): uniform in (0, 1)."""
    k = k or c["k"]
    rng = np.random.default_rng(seed)
    return (rng.random((c["n"], k), np.float32) + np.float32(FLT_MIN), rng.random((c["m"], k), np.float32) + np.float32(FLT_MIN))


def _sweep_problems(c):
    return [k for k in range(c["k"], c["kmax"] + 1) for _ in range(c["restarts"])]


def _consensus_labels(c, seed):
    """Labels of every restart: a planted class per sample, a fifth of them moved at random in each restart."""
    rng = np.random.default_rng(seed)
    m, k, runs = c["m"], c["k"], c["restarts"]
    planted = rng.integers(0, k, m)
    moved = rng.random((runs, m)) < 0.2
    return np.where(moved, rng.integers(0, k, (runs, m)), planted[None, :])


class _Factor:
    """A context's device factor for torch (zero copy); keeps the context alive."""

    def __init__(self, engine, ptr, rows, k, ld):
        self.engine = engine
        self.__cuda_array_interface__ = {"shape": (rows, k), "strides": (4 * ld, 4), "typestr": "<f4", "data": (ptr, False), "version": 3}


def _views(e):
    dW, dH, ld = e.device_factors()
    return (torch.as_tensor(_Factor(e, dW, e.n, e.k, ld), device="cuda"), torch.as_tensor(_Factor(e, dH, e.m, e.k, ld), device="cuda"))


# ---- the cases ---------------------------------------------------------------

def prepare(case, seed):
    c = case
    if c["kind"] in ("run", "step"):
        V = _matrix(c, seed)
        W, H = _factors(c, seed)
        e = nmf.NMF(c["n"], c["m"], c["k"], arm=c["arm"])
        torch.cuda.synchronize()
        e.set_V_device(V.data_ptr(), V.stride(0))
        e.set_WH(W, H)
        e.synchronize()
        return {"case": c, "engine": e, "factors": _views(e)}
    if c["kind"] == "noalloc":
        V = _matrix(c, seed)
        W, H = (torch.from_numpy(x).cuda() for x in _factors(c, seed))
        return {"case": c, "V": V, "W": W, "H": H}
    if c["kind"] == "sweep":
        V = _matrix(c, seed).cpu().numpy()
        ranks = _sweep_problems(c)
        b = nmf.Batch(c["n"], c["m"], ranks)
        b.set_V(V)
        for p, k in enumerate(ranks):
            b.set_WH(p, *_factors(c, seed + 1000 * p, k))
        return {"case": c, "batch": b}
    if c["kind"] == "consensus":
        # restarts whose H assigns each sample to its label with a wide margin: one iteration on a constant
        # matrix scales each row of H and leaves its order
        labels = _consensus_labels(c, seed)
        n, m, k = 32, c["m"], c["k"]
        b = nmf.Batch(n, m, [k] * c["restarts"])
        b.set_V(np.ones((n, m), np.float32))
        W = np.full((n, k), 0.5, np.float32)
        for p in range(c["restarts"]):
            H = np.full((m, k), 0.1, np.float32)
            H[np.arange(m), labels[p]] = 1.0
            b.set_WH(p, W, H)
        b.run(1, 1, 40)
        return {"case": c, "batch": b}
    return {"case": c, "V": _matrix(c, seed).cpu().numpy(), "seed": seed % 1000 + 1}


def run(state):
    c = state["case"]
    if c["kind"] == "run":
        it, conv = state["engine"].run(c["iters"], J, 40)
        W, H = state["factors"]
        return {"W": W, "H": H, "iterations": it, "converged": conv}
    if c["kind"] == "step":
        e = state["engine"]
        e.update_H()
        e.update_W()
        W, H = state["factors"]
        return {"kl": e.kl_divergence(), "W": W, "H": H}
    if c["kind"] == "noalloc":
        V, W, H = state["V"], state["W"], state["H"]
        nmf.update_H_noalloc(V.data_ptr(), V.stride(0), W.data_ptr(), W.stride(0), H.data_ptr(), H.stride(0),
                             c["n"], c["m"], c["k"], torch.cuda.current_stream().cuda_stream)
        return H
    if c["kind"] == "sweep":
        b = state["batch"]
        it, conv = b.run(c["iters"], J, 40)
        ranks, r = _sweep_problems(c), c["restarts"]
        out = {"iterations": it, "converged": conv}
        for k in range(c["k"], c["kmax"] + 1):
            mine = [p for p, q in enumerate(ranks) if q == k]
            out["W%d" % k] = b.W(mine[0])
            out["H%d" % k] = np.stack([b.H(p) for p in mine])
        return out
    if c["kind"] == "consensus":
        counts, nruns, coph = state["batch"].consensus(c["k"])
        return {"counts": counts, "nruns": nruns, "cophenetic": coph}
    W, H, it, conv, distance = nmf.nmf_gpu(state["V"], c["k"], c["iters"], J, 40, state["seed"])
    return {"W": W, "H": H, "iterations": it, "converged": conv, "distance": distance}


# ---- what a pass cannot do without --------------------------------------------

def work(case):
    c = case
    if c["kind"] == "consensus":
        m = c["m"]
        return {"bytes": 4.0 * c["restarts"] * m + 4.0 * m * m + 12.0, "flops": 2.0 * c["restarts"] * m * m + 3.0 * m * m}
    n, m, k = c["n"], c["m"], c["k"]
    factors = 4.0 * (n + m) * k
    if c["kind"] == "run":
        # each half-iteration depends on the other: V is read twice an iteration
        return {"bytes": c["iters"] * (8.0 * n * m + 2 * factors), "flops": c["iters"] * 8.0 * n * m * k}
    if c["kind"] == "step":
        return {"bytes": 3 * 4.0 * n * m + 3 * factors, "flops": 10.0 * n * m * k}
    if c["kind"] == "noalloc":
        return {"bytes": 4.0 * n * m + factors + 4.0 * m * k, "flops": 4.0 * n * m * k}
    if c["kind"] == "sweep":
        ranks = _sweep_problems(c)
        return {"bytes": 4.0 * n * m + 2 * sum(4.0 * (n + m) * q for q in ranks), "flops": c["iters"] * sum(8.0 * n * m * q for q in ranks)}
    return {"bytes": 4.0 * n * m + c["iters"] * (8.0 * n * m + 2 * factors), "flops": (c["iters"] * 8.0 + 2.0) * n * m * k}


# ---- the same in 64 bits --------------------------------------------------------

def _update_H(V, W, H):
    return H * ((V / (W @ H.T)).T @ W) / W.sum(0)


def _update_W(V, W, H):
    return W * ((V / (W @ H.T)) @ H) / H.sum(0)


def _loop(V, W, H, iters):
    for i in range(iters):
        H = _update_H(V, W, H)
        W = _update_W(V, W, H)
        if (i + 1) % J == 0:
            W, H = W.clamp_min(FLT_MIN), H.clamp_min(FLT_MIN)
    return W, H


def _kl(V, WH):
    return torch.where(V > 0, V * torch.log(torch.where(V > 0, V / WH, 1.0)), 0.0).sub_(V).add_(WH).sum().item()


def _c_random(seed, count):
    """The C library's random() after srandom(seed), as FP32 in (0, 1]."""
    libc = ctypes.CDLL(None)
    libc.random.restype = ctypes.c_long
    libc.srandom(ctypes.c_uint(seed))
    draws = np.array([libc.random() for _ in range(count)], np.int64).astype(np.float32)
    return draws / np.float32(2147483647) + np.float32(FLT_MIN)


def _cophenetic(counts, runs):
    """Correlation of 1 - counts / runs with the heights of its average-linkage tree (lowest pair of slots first on ties)."""
    m = counts.shape[0]
    D = 1.0 - counts.astype(np.float64) / runs
    np.fill_diagonal(D, 0.0)
    left = D.copy()
    left[np.tril_indices(m)] = np.inf
    full, size, members = D.copy(), np.ones(m), [[i] for i in range(m)]
    coph = np.zeros((m, m))
    for _ in range(m - 1):
        a, b = divmod(int(np.argmin(left)), m)
        h = left[a, b]
        coph[np.ix_(members[a], members[b])] = h
        coph[np.ix_(members[b], members[a])] = h
        row = (size[a] * full[a] + size[b] * full[b]) / (size[a] + size[b])
        members[a] += members[b]
        members[b] = []
        size[a] += size[b]
        size[b] = 0
        full[a], full[:, a] = row, row
        alive = size > 0
        idx = np.arange(m)
        left[a, :] = np.where((idx > a) & alive, row, np.inf)
        left[:, a] = np.where((idx < a) & alive, row, np.inf)
        left[b, :] = left[:, b] = np.inf
    up = np.triu_indices(m, 1)
    x, y = D[up] - D[up].mean(), coph[up] - coph[up].mean()
    xx, yy = float(x @ x), float(y @ y)
    return float(x @ y) / math.sqrt(xx * yy) if xx > 0 and yy > 0 else 0.0


def exact(case, seed):
    c = case
    if c["kind"] == "consensus":
        labels = _consensus_labels(c, seed)
        counts = (labels[:, :, None] == labels[:, None, :]).sum(0)
        return {"counts": None, "nruns": None, "cophenetic": _cophenetic(counts, c["restarts"])}
    V32 = _matrix(c, seed)
    V = V32.double()
    if c["kind"] == "solve":
        n, m, k = c["n"], c["m"], c["k"]
        x = torch.from_numpy(_c_random(seed % 1000 + 1, (n + m) * k)).cuda().double()
        W, H = _loop(V, x[: n * k].reshape(n, k), x[n * k:].reshape(m, k), c["iters"])
        distance = ((V - W @ H.T).norm() / V.norm()).item()
        return {"W": W, "H": H, "iterations": None, "converged": None, "distance": distance}
    if c["kind"] == "sweep":
        got, out = {}, {"iterations": None, "converged": None}
        for p, k in enumerate(_sweep_problems(c)):
            W, H = (torch.from_numpy(x).cuda().double() for x in _factors(c, seed + 1000 * p, k))
            got.setdefault(k, []).append(_loop(V, W, H, c["iters"]))
        for k, pairs in got.items():
            out["W%d" % k] = pairs[0][0]
            out["H%d" % k] = torch.stack([h for _, h in pairs])
        return out
    W, H = (torch.from_numpy(x).cuda().double() for x in _factors(c, seed))
    if c["kind"] == "run":
        W, H = _loop(V, W, H, c["iters"])
        return {"W": W, "H": H, "iterations": None, "converged": None}
    H = _update_H(V, W, H)
    if c["kind"] == "noalloc":
        return H
    W = _update_W(V, W, H)
    return {"kl": _kl(V, W @ H.T), "W": W, "H": H}
