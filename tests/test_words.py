"""The factored engine's word transforms (csrc/bdc_words.cuh): the identity
they rest on, restated on the CPU, and the engine at the edges of their
ranges against the count engine."""
from math import comb

import numpy as np
import pytest


def _occurrences(x, nx, y, ny):
    d = [1] + [0] * ny
    for i in range(nx):
        c = (x >> (nx - 1 - i)) & 1
        for j in range(ny, 0, -1):
            if ((y >> (ny - j)) & 1) == c:
                d[j] += d[j - 1]
    return d[ny]


def _word_vector(lnq, k, chars, half):
    """c_w: the characters of w consumed on ln q, then the weight of each
    length (the word belongs to a half of `half` characters)."""
    c = {(k, z): lnq[z] for z in range(1 << k)}
    for i, b in enumerate(chars, 1):
        new = {(l, z): c.get((l, z), 0.0) + c[(l + 1, (b << l) | z)] for l in range(k - i, k) for z in range(1 << l)}
        c.update(new)
    return {(l, z): v / comb(half - (k - l), len(chars) - (k - l)) for (l, z), v in c.items()}


@pytest.mark.parametrize("n,k", [(2, 1), (3, 2), (5, 4), (7, 1), (7, 4), (8, 4), (9, 2), (9, 6), (9, 8)])
def test_words_of_one_length_carry_every_split_term(n, k):
    """sum_y N(x, y) ln q(y) from the words of length a of x_hi and b of x_lo
    alone equals the sum over every split point."""
    n1 = (n + 1) // 2
    n2, a = n - n1, k // 2
    b = k - 1 - a
    rev = lambda v, m: int(format(v, f"0{m}b")[::-1], 2) if m else 0  # noqa: E731
    lnq = -np.random.default_rng(n * 32 + k).random(1 << k)
    lnq = np.array([lnq[min(y, rev(y, k))] for y in range(1 << k)])

    def transform(w, words, half, x, other):
        c = _word_vector(lnq, k, [(w >> (words - 1 - i)) & 1 for i in range(words)], half)
        return sum(v * _occurrences(x, other, z, l) for (l, z), v in c.items() if l <= other)

    for x in range(0, 1 << n, max(1, (1 << n) // 24)):
        xh, xl = x >> n2, x & ((1 << n2) - 1)
        got = sum(_occurrences(xh, n1, w, a) * transform(w, a, n1, xl, n2) for w in range(1 << a))
        got += sum(_occurrences(xl, n2, w, b) * transform(rev(w, b), b, n2, rev(xh, n1), n1) for w in range(1 << b))
        want = sum(_occurrences(x, n, y, k) * lnq[y] for y in range(1 << k))
        assert abs(got - want) <= 1e-13 * abs(want)


# the smallest halves, words of no character, odd n, the longest words, and
# strings cut into several slices (more than 11 characters, 12 above k = 12)
EDGES = [(2, 1), (3, 1), (3, 2), (4, 3), (13, 1), (13, 12), (16, 13), (21, 13), (24, 2), (25, 5), (26, 14)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", EDGES)
def test_iteration_at_the_edges_matches_the_count_engine(bdc, n, k):
    """One iteration from a Dirichlet start.  Every sum has terms of one sign
    and fewer than 2^10 roundings on a path, so D (below 10 nats) is off by
    at most 1e-12 and p by as much relative."""
    rng = np.random.default_rng(n * 32 + k)
    out = []
    for engine in ("count", "factored"):
        with bdc.Engine(n, k, engine=engine) as E:
            p0 = rng.exponential(size=E.R) if not out else p0
            E.set_p(p0 / (4.0 * p0.sum()))
            st = E.iterate(1)
            out.append((E.get_p(), st))
    np.testing.assert_allclose(out[1][0], out[0][0], rtol=2e-12, atol=0)
    for key in ("upper_bound", "rate", "lse"):
        assert abs(out[1][1][key] - out[0][1][key]) < 2e-12, key


@pytest.mark.gpu
@pytest.mark.parametrize("n,k,world", [(9, 4, 3), (15, 8, 2), (21, 9, 2)])
def test_shard_sums_and_update_match_the_whole(bdc, n, k, world):
    """Row windows that cut the transforms' slices: the ranks' raw sums add up
    to the count engine's, and their iterates to one engine's."""
    rng = np.random.default_rng(n)
    with bdc.Engine(n, k, engine="count") as E:
        p0 = rng.exponential(size=E.R)
        p0 /= 4.0 * p0.sum()
        E.set_p(p0)
        want = E.shard_q(0, E.R)
    with bdc.Engine(n, k, engine="factored") as E:
        E.set_p(p0)
        E.iterate(1)
        whole = E.get_p()
    shards = [bdc.Engine(n, k, engine="factored", shard=(r, world)) for r in range(world)]
    for E in shards:
        E.set_p(p0)
    acc = [E.fshard_q() for E in shards]
    np.testing.assert_allclose(sum(acc), want, rtol=2e-12, atol=0)
    part = np.array([E.fshard_d(sum(acc)) for E in shards])
    comb5 = np.array([part[:, 0].max(), part[:, 1].sum(), part[:, 2].max(), part[:, 3].sum(), part[:, 4].max()])
    got = []
    for E in shards:
        E.fshard_finish(comb5)
        got.append(E.fshard_get_p())
        E.close()
    np.testing.assert_allclose(np.concatenate(got), whole, rtol=2e-12, atol=0)
