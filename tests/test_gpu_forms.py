"""The forms counted from one build of a root's rows (4-wheel and neighbourhood
statistics): pairs on the same graph share their roots' rows, so every mix of
them, repeated pairs and shards must give each pair's own count, in every tier
and for rows wider than the strip-counted ones."""
import numpy as np
import pytest

import beep_b200 as B
from beep_b200 import patterns as P
from oracle import pyoracle as O
from oracle import synth

pytestmark = pytest.mark.gpu

PATS = P.central_patterns(4) + P.central_patterns(5)
FORMS = [12, 9, 10, 11, 13, 6, 7]  # the 4-wheel, then forms 3, 4, 5, 6, 1, 2


def hubs(n, p, seed, n_hubs=3):
    rng = np.random.default_rng(seed)
    m = int(p * n * (n - 1) / 2)
    us = [rng.integers(0, n, m)] + [np.full(n, n + h) for h in range(n_hubs)]
    vs = [rng.integers(0, n, m)] + [np.arange(n) for _ in range(n_hubs)]
    return synth.to_csr(n + n_hubs, np.concatenate(us), np.concatenate(vs))


GRAPHS = {"small": synth.erdos_renyi(200, 0.2, 1), "thread": hubs(200, 0.08, 2), "warp": hubs(700, 0.02, 3),
          "large": hubs(1500, 0.008, 4), "power": synth.chung_lu(2500, 16.0, 2.1, 5)}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_mixes_match_each_pair_alone(ctx, name):
    rp, col = GRAPHS[name]
    g = B.Graph.from_csr(ctx, rp, col)
    exp = {i: O.count(rp, col, PATS[i], apply_root_cap=False)["count"] for i in FORMS}
    for i in FORMS:
        assert B.count(g, PATS[i]) == exp[i], i
        assert B.count(g, PATS[i], B.SGM, B.OPT_NO_NBHD) == exp[i], i
        assert B.count(g, PATS[i], B.SGM, B.OPT_NO_VIEW_CACHE) == exp[i], i
        assert sum(B.count_shard(g, PATS[i], r, 4) for r in range(4)) == exp[i], i
    for mix in (FORMS, FORMS[::-1], [11, 13], [13, 12, 13], [9, 11, 9, 12, 14, 3], [10, 1, 2, 8, 11]):
        b = B.Batch(ctx)
        for i in mix:
            b.add(g, PATS[i])
        want = [exp[i] if i in exp else B.count(g, PATS[i]) for i in mix]
        got, st = b.run(B.OPT_NO_GRAPH, stats=True)
        assert got == want, mix
        assert st["roots"] > 0
        assert b.run() == want, mix  # captured
        assert b.run() == want, mix
        b.close()
    g.close()


def test_shards_match_oracle(ctx):
    rp, col = GRAPHS["power"]
    g = B.Graph.from_csr(ctx, rp, col)
    for i in FORMS:
        for r in range(3):
            exp = O.count(rp, col, PATS[i], apply_root_cap=False, root_mod=3, root_rem=r)["count"]
            assert B.count_shard(g, PATS[i], r, 3) == exp, (i, r)
    g.close()


def test_rows_wider_than_strips(ctx):
    """Hubs of 16,500: the word-list kernels, mixed with narrower roots."""
    rp, col = hubs(16500, 0.0004, 6, n_hubs=2)
    g = B.Graph.from_csr(ctx, rp, col)
    alone = [B.count(g, PATS[i]) for i in FORMS]
    b = B.Batch(ctx)
    for i in FORMS:
        b.add(g, PATS[i])
    assert b.run() == alone
    for i in (12, 11, 13):  # the 4-wheel, the paw, the diamond
        assert alone[FORMS.index(i)] == O.count(rp, col, PATS[i], apply_root_cap=False)["count"], i
    for i, c in zip(FORMS[1:3], alone[1:3]):
        assert B.count(g, PATS[i], B.SGM, B.OPT_NO_NBHD) == c > 0, i
    b.close()
    g.close()
