"""The single passes and the adjoint on handles with products (ln q, D, the
rate and dI/dp by the factored kernels) against the count engine."""
import numpy as np
import pytest

SIZES = [(13, 12), (16, 13), (19, 9), (20, 10), (21, 13), (25, 5)]


def _start(R, seed):
    rng = np.random.default_rng(seed)
    p = rng.exponential(size=R)
    p[rng.random(R) < 0.05] = 0.0
    return p / (4.0 * p.sum())


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", SIZES)
@pytest.mark.parametrize("iters", [0, 3])
def test_passes_match_the_count_engine(bdc, n, k, iters):
    """At a loaded start with exact zeros and after iterations: sums of one
    sign in FP64, values below 16 nats, errors below 1e-12."""
    out = []
    for engine in ("count", "factored"):
        with bdc.Engine(n, k, engine=engine) as E:
            E.set_p(_start(E.R, n * 32 + k))
            if iters:
                E.iterate(iters)
            lnq = E.log_q()
            other = np.where(lnq != 0.0, lnq * (1.0 + 0.1 * np.cos(np.arange(len(lnq)))), 0.0)
            out.append((lnq, E.log_w(lnq), E.divergence(other), E.divergence(), np.array([E.rate()]), E.get_p()))
    for i, (c, f) in enumerate(zip(*out)):
        np.testing.assert_allclose(f, c, rtol=3e-12, atol=0 if i == 5 else 3e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", SIZES)
def test_adjoint_leaves_the_iterate_as_a_fresh_load(bdc, n, k):
    """I and dI/dp match the count engine's, and later iterations are those of
    the same p loaded anew, whatever ran before."""
    p0 = None
    with bdc.Engine(n, k, engine="count") as C, bdc.Engine(n, k, engine="factored") as E, \
            bdc.Engine(n, k, engine="factored") as G:
        p0 = _start(E.R, n + k)
        for before in (0, 2):
            for h in (C, E, G):
                h.set_p(p0)
                if before:
                    h.iterate(before)
            assert abs(E.mi_forward() - C.mi_forward()) < 3e-12
            np.testing.assert_allclose(E.mi_backward(), C.mi_backward(), rtol=3e-12, atol=3e-12)
            G.set_p(G.get_p())
            a, b = E.iterate(2), G.iterate(2)
            assert a["total_iters"] == b["total_iters"] == 2
            np.testing.assert_allclose(E.get_p(), G.get_p(), rtol=3e-12, atol=0)
            assert abs(a["best_rate"] - b["best_rate"]) < 3e-12
