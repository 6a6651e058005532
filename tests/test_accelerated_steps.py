"""The accelerated loop's steps against the same loop written out on the CPU
oracle: odd and even lengths (a representative's column paired with one that
is none), restarts, and a start so uneven that the extrapolated point leaves
the range in which exp needs no shift."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LN2 = np.log(2.0)


def _loop(O, n, k, p, evals, eta=1.5):
    reps = O.canonicals(n)
    w = O.orbits_of(reps, n).astype(float)

    def lse(v):
        m = v.max()
        return m + np.log(np.sum(w * np.exp(v - m)))

    def evaluate(ly):
        ly = ly - lse(ly)
        py = np.exp(ly)
        lnq = O.log_q(n, k, py, reps)
        d = O.kl(n, k, lnq, reps)
        return d, O.rate(n, k, lnq, py, reps), d.max()

    d, rate, ub = evaluate(np.log(p))
    best_r, best_u = rate, ub
    x = np.log(p) + d
    x -= lse(x)
    y, old, t, prev, far = x, x, 0, -np.inf, False
    for _ in range(evals - 1):
        far = far or abs(y.max()) > 40.0
        d, rate, ub = evaluate(y)
        best_r, best_u = max(best_r, rate), min(best_u, ub)
        if rate >= prev:
            prev, t, old = rate, t + 1, x
            x = y + eta * d
            x = x - lse(x)
            y = x + t / (t + 3.0) * (x - old)
        else:
            prev, t, y = -np.inf, 0, x
    return best_r / LN2, best_u / LN2, far


@pytest.mark.parametrize("n,k,kind", [(4, 2, "even"), (7, 3, "even"), (12, 6, "even"), (13, 6, "even"),
                                      (11, 10, "even"), (10, 5, "uneven"), (13, 7, "uneven")])
def test_steps_match_the_loop_on_the_oracle(bdc, O, n, k, kind):
    from bdc_b200 import dist
    p = dist.dirichlet_start(n, 0.6, 3)
    w = O.orbits_of(O.canonicals(n), n).astype(float)
    if kind == "uneven":
        p = np.full(len(p), 1e-300)
        p[len(p) // 2] = 1.0
    p = p / np.sum(w * p)
    evals = 25
    r, u, far = _loop(O, n, k, p, evals)
    assert far == (kind == "uneven" and n == 13)
    with bdc.Engine(n, k, engine="factored") as E:
        E.set_p(p)
        st = E.accelerate(evals, 1e-300)
    assert st["iters"] == evals
    # 25 steps multiply the rounding of logarithms up to ~300 in size by a
    # growth of a few a step at most
    assert abs(st["best_rate"] - r) < 1e-9 and abs(st["best_upper_bound"] - u) < 1e-9
