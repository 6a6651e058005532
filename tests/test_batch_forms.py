"""Batches of small problems: instances that share the SMs by the direct
iteration, and those that take the products beside one another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# fewer CTAs an instance than alone, down to one; two, and more, of a problem
# that holds both forms; both kinds and a handle with products alone together
@pytest.mark.parametrize("mix", [[(14, 7)] * 3, [(16, 8)] * 40, [(18, 9)] * 2, [(18, 9)] * 3, [(20, 3)] * 4,
                                 [(10, 5), (17, 10), (17, 9), (13, 11)]])
def test_batch_matches_single_handles(bdc, mix):
    """Iterations and accelerated steps of a batch against the same handles
    alone.  The sums are of one sign; they are taken in another order, which
    moves an iterate by a few times 1e-16 a step, and the 17 steps multiply that
    by at most 1e3."""
    rng = np.random.default_rng(len(mix) * 64 + mix[0][0])
    E = [bdc.Engine(n, k, engine="factored") for n, k in mix]
    try:
        p0 = [rng.exponential(size=e.R) for e in E]
        p0 = [v / (4.0 * v.sum()) for v in p0]
        def load():
            for e, p in zip(E, p0):
                e.set_p(p)
        with bdc.Batch(E) as B:
            load()
            it = B.iterate(19)
            p_it = [e.get_p() for e in E]
            load()
            acc, _ = B.accelerate(16, 0.0)
            p_acc = [e.get_p() for e in E]
        load()
        for e, st, p in zip(E, it, p_it):
            one = e.iterate(19)
            assert one["iters"] == st["iters"] == 19
            np.testing.assert_allclose(p, e.get_p(), rtol=1e-12, atol=0)
            assert abs(one["upper_bound"] - st["upper_bound"]) < 1e-12
        load()
        for e, st, p in zip(E, acc, p_acc):
            one = e.accelerate(st["iters"], 0.0)  # (a batch's evaluations come in graphs of 8 after the first)
            assert one["iters"] == st["iters"] == 17
            np.testing.assert_allclose(p, e.get_p(), rtol=1e-12, atol=0)
            assert abs(one["best_rate"] - st["best_rate"]) < 1e-12
    finally:
        for e in E:
            e.close()
