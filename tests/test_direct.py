"""The direct iteration of small problems (csrc/bdc_direct.cuh): every lane
layout, one CTA and several, against the count engine."""
import numpy as np
import pytest

# one piece a row up to 34 (k = 10); one CTA, several, and the most; the last
# sizes on either side of the rule (16-bit entries, k <= 10)
SIZES = [(5, 2), (9, 4), (16, 4), (20, 4), (10, 5), (15, 5), (11, 6), (18, 6), (10, 7), (16, 7), (12, 8), (15, 8),
         (11, 9), (17, 9), (13, 10), (18, 10), (16, 11), (19, 8)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", SIZES)
def test_chain_matches_the_count_engine(bdc, n, k):
    """Chains of 1, 9 and 3 iterations in a row, and the zeros of the start.
    An iteration multiplies the relative error of p by at most 1 + 1e-12 on
    top of 1e-12 of its own (sums of one sign, values below 16 nats)."""
    rng = np.random.default_rng(n * 16 + k)
    out = []
    for engine in ("count", "factored"):
        with bdc.Engine(n, k, engine=engine) as E:
            if not out:
                p0 = rng.exponential(size=E.R)
                p0[rng.random(E.R) < 0.1] = 0.0
                p0 /= 4.0 * p0.sum()
            E.set_p(p0)
            st = [E.iterate(m) for m in (1, 9, 3)]
            out.append((E.get_p(), st))
    (pc, sc), (pf, sf) = out
    np.testing.assert_allclose(pf, pc, rtol=3e-11, atol=0)
    for a, b in zip(sc, sf):
        assert a["iters"] == b["iters"] and a["total_iters"] == b["total_iters"]
        for key in ("upper_bound", "rate", "lse", "best_upper_bound", "best_rate"):
            assert abs(a[key] - b[key]) < 3e-11, key


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(10, 5), (15, 8)])
def test_chain_stops_at_its_threshold(bdc, n, k):
    """The stop fires inside a chain: the same iteration as the count engine,
    and nothing moves afterwards."""
    got = []
    for engine in ("count", "factored"):
        with bdc.Engine(n, k, engine=engine) as E:
            E.set_uniform()
            st = E.iterate(500, 0.02)
            p = E.get_p()
            got.append((st["iters"], st["mx"], p))
            assert st["converged"] and 1 < st["iters"] < 500
    assert got[0][0] == got[1][0]
    assert abs(got[0][1] - got[1][1]) < 1e-10
    np.testing.assert_allclose(got[1][2], got[0][2], rtol=1e-10, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(10, 5), (14, 7)])
def test_batch_and_rescale_on_direct_handles(bdc, n, k):
    """A batch of direct handles equals the handles alone, and a start scaled
    out of the exponential's range recovers."""
    rng = np.random.default_rng(3)
    E = [bdc.Engine(n, k, engine="factored") for _ in range(3)]
    p0 = [rng.exponential(size=E[0].R) for _ in range(2)]
    p0 = [v / (4.0 * v.sum()) for v in p0]
    E[0].set_p(p0[0])
    E[1].set_p(p0[1] * 1e-280)
    B = bdc.Batch(E[:2])
    B.iterate(20)
    for i, scale in ((0, 1.0), (1, 1e-280)):
        E[2].set_p(p0[i] * scale)
        E[2].iterate(20)
        np.testing.assert_allclose(E[i].get_p(), E[2].get_p(), rtol=1e-12, atol=0)
    B.close()
    for e in E:
        e.close()
