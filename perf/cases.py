"""Timed cases of the Blahut-Arimoto engine, through its Python entry points.

A case is one call, or the short run of calls, that a program makes with a
handle that it keeps and a starting distribution of its own: plain iterations,
the reference-shaped host step, the single passes of the reference's host API,
the adjoint, the accelerated loop, the certified solver and a batch.  Sizes are
those of the repository's own configurations, tests and benchmark.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "bdc-upper-bounds-gpu_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import bdc_b200  # noqa: E402

# sizes of the batched benchmark, one instance each
BATCH_MIX = "16/8,18/6,20/10,22/11,24/8"


def listed():
    return [
        # a small problem run to convergence in chunks: latency and launches
        {"name": "iterate_10_5", "op": "iterate", "n": 10, "k": 5, "engine": "auto", "iters": 64, "zeros": 0.0},
        # an odd n, where the two halves of a string differ in length
        {"name": "iterate_17_9", "op": "iterate", "n": 17, "k": 9, "engine": "auto", "iters": 64, "zeros": 0.0},
        # the ordinary size
        {"name": "iterate_20_10", "op": "iterate", "n": 20, "k": 10, "engine": "auto", "iters": 64, "zeros": 0.0},
        # the headline size of the benchmark
        {"name": "iterate_24_12", "op": "iterate", "n": 24, "k": 12, "engine": "auto", "iters": 32, "zeros": 0.0},
        # the largest problem that one GPU is used for
        {"name": "iterate_28_13", "op": "iterate", "n": 28, "k": 13, "engine": "auto", "iters": 4, "zeros": 0.0},
        # the exact-count engine, which a user asks for by name
        {"name": "count_20_10", "op": "iterate", "n": 20, "k": 10, "engine": "count", "iters": 8, "zeros": 0.0},
        # the drop-in step: host vector in, host vector out, as the reference's loop calls it
        {"name": "host_step_24_12", "op": "host_step", "n": 24, "k": 12},
        # the reference's single passes: ln q, ln p + D and the rate of one distribution
        {"name": "passes_20_10", "op": "passes", "n": 20, "k": 10},
        # forward and backward of I(p;W) for an optimiser that keeps p on the device
        {"name": "adjoint_26_13", "op": "adjoint", "n": 26, "k": 13},
        # the momentum loop of the accelerated method at the headline size
        {"name": "accelerate_24_12", "op": "accelerate", "n": 24, "k": 12, "evals": 64},
        # the time to a certified bracket, from a start near the uniform one
        {"name": "solve_20_10", "op": "solve", "n": 20, "k": 10, "jitter": 0.5},
        # several problems of different sizes together
        {"name": "batch_mixed", "op": "batch", "mix": BATCH_MIX, "iters": 32},
    ]


def draw(rng):
    op = rng.choice(["iterate", "iterate", "iterate", "iterate", "count", "host_step", "passes", "adjoint",
                     "accelerate", "solve", "batch"])
    if op == "iterate":
        n = rng.randint(8, 27)
        k = rng.randint(2, min(13, n - 1))
        most = max(2, min(96, 1 << max(0, 28 - n)))
        return {"op": "iterate", "n": n, "k": k, "engine": "auto", "iters": rng.randint(max(2, most // 4), most),
                "zeros": rng.choice([0.0, 0.0, 0.1])}
    if op == "count":
        n = rng.randint(9, 22)
        k = rng.randint(2, min(n, 31 - n, 12))
        return {"op": "iterate", "n": n, "k": k, "engine": rng.choice(["count", "count", "count-fp32c"]),
                "iters": rng.randint(3, 8), "zeros": 0.0}
    if op == "host_step":
        n = rng.randint(9, 24)
        return {"op": "host_step", "n": n, "k": rng.randint(3, min(12, n - 1))}
    if op == "passes":
        n = rng.randint(9, 22)
        return {"op": "passes", "n": n, "k": rng.randint(3, min(n - 1, 11))}
    if op == "adjoint":
        n = rng.randint(10, 25)
        return {"op": "adjoint", "n": n, "k": rng.randint(4, min(12, n - 1))}
    if op == "accelerate":
        n = rng.randint(10, 24)
        return {"op": "accelerate", "n": n, "k": rng.randint(4, min(12, n - 2)), "evals": rng.randint(24, 64)}
    if op == "solve":
        n = rng.randint(8, 10) * 2
        return {"op": "solve", "n": n, "k": n // 2, "jitter": rng.uniform(0.2, 0.6)}
    sizes = []
    for _ in range(rng.randint(2, 5)):
        n = rng.randint(12, 22)
        sizes.append(f"{n}/{rng.randint(4, min(11, n - 2))}")
    return {"op": "batch", "mix": ",".join(sizes), "iters": rng.randint(8, 32)}


# ------------------------------------------------------------------ inputs
def _reverse(x, n):
    r = torch.zeros_like(x)
    for i in range(n):
        r |= ((x >> i) & 1) << (n - 1 - i)
    return r


def _representatives(n):
    """(representatives ascending, orbit sizes) on the GPU, by their definition."""
    x = torch.arange(1 << (n - 1), device="cuda", dtype=torch.int64)  # the top bit of a representative is 0
    rv = _reverse(x, n)
    rc = _reverse(x ^ ((1 << n) - 1), n)
    keep = (x <= rv) & (x <= rc)
    x, rv, rc = x[keep], rv[keep], rc[keep]
    return x, torch.where((x == rv) | (x == rc), 2.0, 4.0).to(torch.float64)


_orbits = {}


def _orbit_sizes(n):
    if n not in _orbits:
        _orbits.clear()
        _orbits[n] = _representatives(n)[1]
    return _orbits[n]


def _start(n, seed, zeros=0.0, jitter=None):
    """A distribution per representative with sum |O| p = 1: the orbit mean of
    a Dirichlet(1) draw over all strings, a share `zeros` of its entries at
    exact 0; or, with `jitter`, the uniform start with each entry moved by up
    to that share."""
    o = _orbit_sizes(n)
    g = torch.Generator(device="cuda").manual_seed(seed)
    if jitter is not None:
        p = 1.0 + jitter * torch.rand(len(o), dtype=torch.float64, device="cuda", generator=g)
    else:
        p = torch.zeros_like(o)
        e = torch.empty_like(o)
        for j in range(4):
            e.exponential_(generator=g)
            p += e if j < 2 else torch.where(o > 2.0, e, 0.0)
        p /= o
        if zeros > 0.0:
            p[torch.rand(len(o), dtype=torch.float64, device="cuda", generator=g) < zeros] = 0.0
    return p / (o * p).sum()


def _mix(case):
    return [tuple(int(v) for v in s.split("/")) for s in case["mix"].split(",")]


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        engines, starts = [], []
        for i, (n, k) in enumerate(_mix(case)):
            engines.append(bdc_b200.Engine(n, k))
            starts.append(_start(n, seed * 64 + i))
        return {"case": case, "engines": engines, "batch": bdc_b200.Batch(engines), "p": starts,
                "out": [torch.empty_like(p) for p in starts]}
    n, k = case["n"], case["k"]
    E = bdc_b200.Engine(n, k, engine=case.get("engine", "auto"))
    p = _start(n, seed, case.get("zeros", 0.0), case.get("jitter"))
    if op in ("host_step", "passes"):
        return {"case": case, "engine": E, "p": p.cpu().numpy()}
    return {"case": case, "engine": E, "p": p, "out": torch.empty_like(p)}


# --------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    op = case["op"]
    if op == "batch":
        for E, p in zip(state["engines"], state["p"]):
            E.set_p_device(p.data_ptr())
        st = state["batch"].iterate(case["iters"])
        for E, out in zip(state["engines"], state["out"]):
            E.get_p_device(out.data_ptr())
        return {"p": state["out"], "upper_bound": [s["upper_bound"] for s in st], "rate": [s["rate"] for s in st]}
    E, p = state["engine"], state["p"]
    if op == "host_step":
        return {"p": E.baa_iteration(p)}
    if op == "passes":
        E.set_p(p)
        lnq = E.log_q()
        return {"lnq": lnq, "logw": E.log_w(lnq), "rate": np.array([E.rate()])}
    out = state["out"]
    E.set_p_device(p.data_ptr())
    if op == "adjoint":
        info = E.mi_forward()
        E.mi_backward_device(out.data_ptr())
        return {"info": np.array([info]), "grad": out}
    if op == "accelerate":
        st = E.accelerate(case["evals"], 0.0)
        keys = ("best_upper_bound", "best_rate")
    elif op == "solve":
        st = E.solve(1e-9, 20000)
        keys = ("best_upper_bound", "best_rate")
    else:
        st = E.iterate(case["iters"])
        keys = ("mx", "upper_bound", "rate", "lse")
    E.get_p_device(out.data_ptr())
    return {"p": out, "stats": np.array([st[key] for key in keys])}


# -------------------------------------------------------------------- work
def _num_reps(n):
    return ((1 << n) + (1 << ((n + 1) // 2)) + ((1 << (n // 2)) if n % 2 == 0 else 0)) // 4


def _contraction(n, k):
    """Length of the stacked contraction of the split identity: 2^min(j, k - j)
    summed over the split points j."""
    n1 = (n + 1) // 2
    n2 = n - n1
    total = 0
    for j in range(max(0, k - n2), min(k, n1) + 1):
        m = k - j
        left = m == n2 or (j != n1 and j <= m)
        total += 1 << (j if left else m)
    return total


def _iteration_work(n, k, engine):
    """(bytes, flops) of one iteration: p and h(x) read, p written; the q pass
    and the D pass, a multiply-add per contraction index and representative
    (per pair of strings on the count path)."""
    R = _num_reps(n)
    per = (1 << k) if engine.startswith("count") or k == n else min(1 << k, _contraction(n, k))
    return 24.0 * R, 4.0 * R * per


def work(case):
    op = case["op"]
    if op == "batch":
        w = [(_num_reps(n), _iteration_work(n, k, "auto")) for n, k in _mix(case)]
        return {"bytes": sum(16.0 * R + case["iters"] * b for R, (b, _) in w),
                "flops": sum(case["iters"] * f for _, (_, f) in w)}
    n, k = case["n"], case["k"]
    R = _num_reps(n)
    b, f = _iteration_work(n, k, case.get("engine", "auto"))
    if op in ("host_step", "passes", "adjoint"):
        # one q pass and one D pass serve every output
        return {"bytes": b, "flops": f}
    if op == "solve":
        # the evaluations that the full space needs, about n^2, set the scale
        return {"bytes": 16.0 * R + n * n * b, "flops": n * n * f}
    its = case["evals"] if op == "accelerate" else case["iters"]
    return {"bytes": 16.0 * R + its * b, "flops": its * f}


# ------------------------------------------------------------------- exact
class _Dense:
    """BA over the dense count matrix N(x, y), exact integers held in FP32 and
    summed in FP64, a block of representatives at a time."""

    def __init__(self, n, k):
        self.n, self.k = n, k
        self.C = float(math.comb(n, k))
        self.x, self.o = _representatives(n)
        ny = 1 << k
        step = max(1, (1 << 27) >> k)
        self.blocks = []
        self.h = torch.empty_like(self.o)
        for a in range(0, len(self.x), step):
            b = min(len(self.x), a + step)
            N = self._counts(self.x[a:b])
            self.h[a:b] = (torch.special.xlogy(N, N).sum(1)) / self.C - math.log(self.C)
            self.blocks.append((a, b, N.to(torch.float32)))
        y = torch.arange(ny, device="cuda", dtype=torch.int64)
        ry = _reverse(y, k)
        self.images = (y, ry, y ^ (ny - 1), ry ^ (ny - 1))
        self.rep_y = torch.stack(self.images).min(0).values

    def _counts(self, x):
        """Subsequence counts by adding one character of x at a time: a word
        of length m ends at the new character or before it."""
        n, k = self.n, self.k
        cnt = [torch.zeros(len(x), 1 << m, dtype=torch.float64, device="cuda") for m in range(k + 1)]
        cnt[0][:] = 1.0
        for i in range(n):
            bit = (x >> (n - 1 - i)) & 1
            on = torch.stack([1.0 - bit.to(torch.float64), bit.to(torch.float64)], 1)  # the word's last character
            for m in range(min(k, i + 1), 0, -1):
                cnt[m].view(len(x), -1, 2).add_(cnt[m - 1].unsqueeze(2) * on.unsqueeze(1))
        return cnt[k]

    def lnq(self, p):
        acc = torch.zeros(1 << self.k, dtype=torch.float64, device="cuda")
        w = self.o * p
        for a, b, N in self.blocks:
            acc += w[a:b] @ N.to(torch.float64)
        q = sum(acc[i] for i in self.images) / (4.0 * self.C)
        return torch.where(q > 0, q.log(), 0.0)

    def divergence(self, lnq):
        D = torch.empty_like(self.h)
        for a, b, N in self.blocks:
            D[a:b] = self.h[a:b] - (N.to(torch.float64) @ lnq) / self.C
        return D

    def iterate(self, p, iters):
        ln2 = math.log(2.0)
        for _ in range(iters):
            D = self.divergence(self.lnq(p))
            lnp = torch.where(p > 0, p.log(), 0.0)  # ln 0 = 0, the reference's rule
            logw = lnp + D
            s = logw.max()
            e = (logw - s).exp()
            lse = s + (self.o * e).sum().log()
            rate = (self.o * p * D).sum()
            mx = math.inf if bool((p == 0).any()) else float((D.max() - lse) / ln2)
            p = (logw - lse).exp()
            stats = [mx, float(D.max() / ln2), float(rate / ln2), float(lse / ln2)]
        return p, stats


def _fits(n, k):
    return _num_reps(n) << k <= 1 << 31


def exact(case, seed):
    op = case["op"]
    if op in ("accelerate", "solve"):
        return None  # paths of many steps with decisions of their own
    if op == "batch":
        ps, ubs, rates = [], [], []
        for i, (n, k) in enumerate(_mix(case)):
            if not _fits(n, k):
                ps.append(None)
                ubs.append(None)
                rates.append(None)
                continue
            p, st = _Dense(n, k).iterate(_start(n, seed * 64 + i), case["iters"])
            ps.append(p)
            ubs.append(st[1])
            rates.append(st[2])
        return {"p": ps, "upper_bound": ubs, "rate": rates}
    n, k = case["n"], case["k"]
    if not _fits(n, k):
        return None
    W = _Dense(n, k)
    p = _start(n, seed, case.get("zeros", 0.0))
    if op == "iterate":
        p, st = W.iterate(p, case["iters"])
        return {"p": p, "stats": np.array(st)}
    if op == "host_step":
        return {"p": W.iterate(p, 1)[0].cpu().numpy()}
    lnq = W.lnq(p)
    D = W.divergence(lnq)
    rate = float((W.o * p * D).sum())
    if op == "adjoint":
        return {"info": np.array([rate]), "grad": W.o * (D - 1.0)}
    y = torch.arange(1 << (k - 1), device="cuda", dtype=torch.int64)
    lnq_slots = torch.where(W.rep_y[: 1 << (k - 1)] == y, lnq[: 1 << (k - 1)], 0.0)
    return {"lnq": lnq_slots.cpu().numpy(), "logw": (p.log() + D).cpu().numpy(), "rate": np.array([rate])}
