"""Queries counted from degrees and triangle counts (stars, the triangle, cones
over one edge, a wedge, two disjoint edges and a three-leaf star) against the
oracle and against the walk (the same call with BEEP_OPT_NO_NBHD), under
several labellings, alone and in batches that share a view, repeat a pair and
mix in pairs that walk."""
import itertools
import random

import numpy as np
import pytest

import beep_b200 as B
from beep_b200 import patterns as P
from oracle import pyoracle as O
from oracle import synth

pytestmark = pytest.mark.gpu

QUERIES = {"wedge": P.WEDGE, "triangle": P.TRIANGLE,
           **{f"c4_{i}": q for i, q in enumerate(P.central_patterns(4)[:3])},
           **{f"c5_{i}": P.central_patterns(5)[i] for i in (0, 1, 2, 3, 4, 5)}}


def relabel(q, seed):
    perm = list(range(max(max(e) for e in q) + 1))
    random.Random(seed).shuffle(perm)
    return sorted({(perm[a], perm[b]) for a, b in q})


def graphs():
    rng = np.random.default_rng(4)
    yield "er", synth.erdos_renyi(700, 0.02, 5)
    yield "sparse", synth.erdos_renyi(2000, 0.0008, 6)  # few triangles, many rows of one entry
    yield "power", synth.chung_lu(1500, 12.0, 2.1, 7)
    yield "dense", synth.erdos_renyi(130, 0.5, 8)
    yield "star", synth.to_csr(70, np.zeros(69, np.int64), np.arange(1, 70))
    yield "one_triangle", synth.to_csr(3, np.array([0, 0, 1]), np.array([1, 2, 2]))
    yield "one_edge", synth.to_csr(2, np.array([0]), np.array([1]))
    # hubs joined to everything: long oriented lists, some of them empty
    n = 1300
    us = [rng.integers(0, n, 4000), np.full(n, n), np.full(n, n + 1), [n]]
    vs = [rng.integers(0, n, 4000), np.arange(n), np.arange(n), [n + 1]]
    yield "hubs", synth.to_csr(n + 2, np.concatenate(us), np.concatenate(vs))


@pytest.mark.parametrize("name,csr", list(graphs()), ids=lambda x: x if isinstance(x, str) else "")
def test_forms_match_oracle_and_walk(ctx, name, csr):
    rp, col = csr
    g = B.Graph.from_csr(ctx, rp, col)
    for qname, q in QUERIES.items():
        exp = O.count(rp, col, q, apply_root_cap=False)["count"] if qname != "wedge" else \
            int((np.diff(rp).astype(np.int64) * (np.diff(rp) - 1) // 2).sum())
        for seed in range(3):
            ql = relabel(q, seed)
            assert B.count(g, ql) == exp, (qname, seed)
            assert B.count(g, ql, B.SGM, B.OPT_NO_NBHD) == exp, (qname, seed)
        if qname != "wedge":
            sgc = O.count(rp, col, q, sgc=True, apply_root_cap=False)["count"]
            assert B.count(g, q, B.SGC) == sgc, qname
        assert sum(B.count_shard(g, q, r, 3) for r in range(3)) == exp, qname
        assert B.count(g, q, B.SGM, B.OPT_TIMING | B.OPT_ALG_BYTES | B.OPT_NO_VIEW_CACHE) == exp, qname
    g.close()


def test_batches_share_views_and_counters(ctx):
    csrs = [c for n, c in graphs() if n in ("er", "power", "one_edge", "hubs")]
    gs = [B.Graph.from_csr(ctx, rp, col) for rp, col in csrs]
    qs = list(QUERIES.values()) + [P.K4, P.W5, P.DIAMOND, P.TRIANGLE, P.K5]
    b = B.Batch(ctx)
    want = []
    for g, (rp, col) in zip(gs, csrs):
        for q in qs:
            b.add(g, q)
            want.append(B.count(g, q, B.SGM, B.OPT_NO_NBHD))
    got, st = b.run(B.OPT_NO_GRAPH, stats=True)
    assert got == want
    assert st["roots"] > 0 and st["overflow_pairs"] == 0
    assert b.run() == want  # captured
    assert b.run() == want
    # a graph dropped and built again, views shared within one call
    for rp, col in csrs:
        g = B.Graph.from_csr(ctx, rp, col)
        bb = B.Batch(ctx)
        for q in (P.K4, P.DIAMOND, P.TAILED_TRIANGLE):
            bb.add(g, q)
        exp = [O.count(rp, col, q, apply_root_cap=False)["count"] for q in (P.K4, P.DIAMOND, P.TAILED_TRIANGLE)]
        assert bb.run(B.OPT_NO_GRAPH) == exp
        bb.close()
        g.close()
    b.close()
    for g in gs:
        g.close()
