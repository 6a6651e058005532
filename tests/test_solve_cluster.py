"""The restricted loop in one thread-block cluster: the point that the solver
returns carries its certified bracket by the other engine's passes, from the
smallest output sets (fewer members than CTAs, output orbits padded to four)
to rows that do not fit the cluster's shared memory (24/12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(4, 1), (6, 2), (9, 4), (11, 5), (15, 8), (20, 10), (21, 11), (24, 12)])
def test_solved_point_carries_its_bracket(bdc, n, k):
    from bdc_b200 import dist
    with bdc.Engine(n, k, engine="factored") as E:
        E.set_p(dist.dirichlet_start(n, 0.8, 5))
        st = E.solve(1e-9, 20000)
        p = E.get_p()
    assert st["converged"] and 0.0 <= st["best_upper_bound"] - st["best_rate"] < 1e-9
    with bdc.Engine(n, k, engine="count") as E:
        E.set_p(p)
        d = E.divergence(E.log_q())
        rate = E.rate()
    # two engines on one point: sums of < 2^20 FP64 terms of size < 20 nats
    assert abs(rate / np.log(2.0) - st["rate"]) < 1e-11
    assert abs(d.max() / np.log(2.0) - st["upper_bound"]) < 1e-11
