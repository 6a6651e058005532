"""The products and word transforms at sizes that the direct iteration does
not take: words of one or no character (one column of each product, tiles of
one row), and the longest words of short halves.  test_words.py's smallest
sizes run the direct iteration."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(22, 1), (23, 1), (22, 2), (23, 2), (12, 11), (13, 11), (15, 14)])
def test_iteration_matches_the_count_engine(bdc, n, k):
    """One iteration from a Dirichlet start.  Every sum has terms of one sign
    and fewer than 2^12 roundings on a path (2^21 representatives, added in
    slices and trees), so D (below 11 nats) is off by at most 1e-11 and p by
    as much relative; the mean error is far less."""
    rng = np.random.default_rng(n * 32 + k)
    out = []
    for engine in ("count", "factored"):
        with bdc.Engine(n, k, engine=engine) as E:
            p0 = rng.exponential(size=E.R) if not out else p0
            E.set_p(p0 / (4.0 * p0.sum()))
            if engine == "factored":
                assert E.profile(1)["main_kind"] != 3
                E.set_p(p0 / (4.0 * p0.sum()))
            st = E.iterate(1)
            out.append((E.get_p(), st))
    np.testing.assert_allclose(out[1][0], out[0][0], rtol=1e-11, atol=0)
    for key in ("upper_bound", "rate", "lse"):
        assert abs(out[1][1][key] - out[0][1][key]) < 1e-11, key
