"""Neighbourhood-statistics forms counted by bit-sliced counters, at the edges
of their words, strips and tiers: the cones over a triangle + isolated vertex,
a 4-path, a paw and a diamond, against the oracle and against the walk."""
import numpy as np
import pytest

import beep_b200 as B
from beep_b200 import patterns as P
from oracle import pyoracle as O
from oracle import synth

pytestmark = pytest.mark.gpu

PATS = P.central_patterns(4) + P.central_patterns(5)


def tower(roots, n, p, seed, twins=True):
    """`roots` roots joined to all of n vertices that carry G(n, p); with
    twins, two of the n are joined to all the others (so that they have n - 2
    common neighbours), and the n outrank roots of the same degree."""
    rng = np.random.default_rng(seed)
    m = int(p * n * (n - 1) / 2)
    us, vs = [rng.integers(0, n, m)], [rng.integers(0, n, m)]
    for t in (0, 1) if twins else ():
        us.append(np.full(n, t))
        vs.append(np.arange(n))
    for r in range(roots):
        us.append(np.full(n, n + r))
        vs.append(np.arange(n))
    return synth.to_csr(n + roots, np.concatenate(us), np.concatenate(vs))


@pytest.mark.parametrize("n,p", [(65, 0.2), (256, 0.05), (257, 0.05), (1023, 0.008), (1024, 0.008), (1025, 0.008),
                                 (2048, 0.002), (2049, 0.002)])
def test_forms_at_the_edges(ctx, n, p):
    rp, col = tower(3, n, p, n)
    g = B.Graph.from_csr(ctx, rp, col)
    for i, form in ((9, 3), (10, 4), (11, 5), (13, 6)):
        assert B.Query.from_edges(PATS[i]).plan()["nbhd"] == form
        exp = O.count(rp, col, PATS[i], apply_root_cap=False)["count"]
        assert B.count(g, PATS[i]) == exp > 0, i
        assert B.count(g, PATS[i], B.SGM, B.OPT_NO_NBHD) == exp, i
    g.close()


def test_wide_rows(ctx):
    """Rows of 16,384 and 16,385 bits: the last strip-counted width and the
    first one counted from word lists."""
    for n in (16384, 16385):
        rp, col = tower(1, n, 0.0005, n, twins=False)
        g = B.Graph.from_csr(ctx, rp, col)
        for i in (9, 10):
            assert B.count(g, PATS[i]) == B.count(g, PATS[i], B.SGM, B.OPT_NO_NBHD) > 0, i
        g.close()
