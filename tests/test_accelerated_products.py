"""The accelerated loop's steps on handles whose iterations run by the
products, against the loop on the CPU oracle: an even and an odd length, and
starts whose extrapolated point leaves the range in which exp needs no shift
(2 and 3 blocks share that pass here)."""
import numpy as np
import pytest

from test_accelerated_steps import _loop

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,kind", [(12, 11, "even"), (13, 11, "even"), (12, 11, "ramp"), (13, 11, "ends")])
def test_steps_match_the_loop_on_the_oracle(bdc, O, n, k, kind):
    from bdc_b200 import dist
    p = dist.dirichlet_start(n, 0.6, 3)
    w = O.orbits_of(O.canonicals(n), n).astype(float)
    at = np.arange(len(p))
    if kind == "ramp":
        p = 10.0 ** (-300.0 * at / len(p))
    elif kind == "ends":
        p = np.where(at % 64 == 0, 1.0, 1e-300)
    p = p / np.sum(w * p)
    evals = 25
    r, u, far = _loop(O, n, k, p, evals)
    assert far == (kind != "even")
    with bdc.Engine(n, k, engine="factored") as E:
        E.set_p(p)
        assert E.profile(1)["main_kind"] != 3
        E.set_p(p)
        st = E.accelerate(evals, 1e-300)
    assert st["iters"] == evals
    # 25 steps multiply the rounding of logarithms up to ~700 in size by a
    # growth of a few a step at most
    assert abs(st["best_rate"] - r) < 1e-9 and abs(st["best_upper_bound"] - u) < 1e-9
