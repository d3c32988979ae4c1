"""Clique counts of every tier: closed forms on complete graphs whose domains
sit at the edges of words, tiers and of the deep walks' split, and the
oracle's clique counter on random graphs."""
import itertools
import math

import numpy as np
import pytest

import beep_b200 as B
from beep_b200 import patterns as P
from oracle import pyoracle as O
from oracle import synth

pytestmark = pytest.mark.gpu


def clique(k):
    return P._undirected(list(itertools.combinations(range(k), 2)))


@pytest.mark.parametrize("n,ks", [
    (9, (4, 5, 6, 7)), (25, (4, 5, 6, 7)), (26, (6, 7, 8)), (33, (4, 5, 6, 7)), (64, (4, 5, 6)), (65, (4, 5, 6, 7)),
    (66, (4, 5, 6, 7)), (97, (4, 5, 6)), (256, (4, 5)), (257, (4, 5)), (258, (4, 5)), (1024, (4,)), (1025, (4,)),
    (1026, (4,))])
def test_complete_graphs(ctx, n, ks):
    iu = np.triu_indices(n, 1)
    rp, col = synth.to_csr(n, iu[0], iu[1])
    g = B.Graph.from_csr(ctx, rp, col)
    for k in ks:
        assert B.count(g, clique(k)) == math.comb(n, k), k
    g.close()


@pytest.mark.parametrize("n,p,seed", [(90, 0.4, 1), (400, 0.3, 2), (900, 0.15, 3)])
def test_random_graphs(ctx, n, p, seed):
    rp, col = synth.erdos_renyi(n, p, seed)
    g = B.Graph.from_csr(ctx, rp, col)
    b = B.Batch(ctx)
    for k in (4, 5, 6, 7):
        b.add(g, clique(k))
    exp = [O.count_cliques(rp, col, k) for k in (4, 5, 6, 7)]
    assert b.run() == exp
    assert b.run() == exp  # the captured launches
    assert [B.count(g, clique(k)) for k in (4, 5, 6, 7)] == exp
    # deep walks that are not cliques are split the same way
    wheel6 = P._undirected([(0, i) for i in range(1, 6)] + [(i, i % 5 + 1) for i in range(1, 6)])
    if n == 90:
        assert B.count(g, wheel6) == O.count(rp, col, wheel6, apply_root_cap=False)["count"]
    b.close()
    g.close()
