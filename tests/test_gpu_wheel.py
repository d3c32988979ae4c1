"""4-wheel counts by bit-sliced counters (medium tier: rows in shared memory,
large tier: strips of 32 words) against the oracle, at the edges of their
words, strips and tiers and with counters that reach the highest slices."""
import numpy as np
import pytest

import beep_b200 as B
from beep_b200 import patterns as P
from oracle import pyoracle as O
from oracle import synth

pytestmark = pytest.mark.gpu


def hub_over(n, p, twins, seed):
    """Hub 0 over n vertices with G(n, p) among them; with twins, the last two
    of the n are joined to all the others, so that they have n - 2 common
    neighbours in the hub's neighbourhood."""
    rng = np.random.default_rng(seed)
    m = int(p * n * (n - 1) / 2)
    us = [np.zeros(n, np.int64), rng.integers(1, n + 1, m)]
    vs = [np.arange(1, n + 1), rng.integers(1, n + 1, m)]
    for t in (n - 1, n) if twins else ():
        us.append(np.full(n - 2, t, np.int64))
        vs.append(np.arange(1, n - 1))
    return synth.to_csr(n + 1, np.concatenate(us), np.concatenate(vs))


@pytest.mark.parametrize("n,p,twins", [
    (64, 0.3, True), (65, 0.3, True), (96, 0.5, False), (255, 0.1, True), (256, 0.1, True), (257, 0.1, True),
    (300, 0.5, False), (1023, 0.01, True), (1024, 0.01, True), (1025, 0.01, True), (2048, 0.004, True),
    (2049, 0.004, True), (16384, 0.0003, True), (16385, 0.0003, True), (16417, 0.0004, True), (33000, 0.0001, True)])
def test_hub_neighbourhoods(ctx, n, p, twins):
    rp, col = hub_over(n, p, twins, n)
    exp = O.count(rp, col, P.W5, apply_root_cap=False)["count"]
    assert exp > 0
    g = B.Graph.from_csr(ctx, rp, col)
    assert B.count(g, P.W5) == exp  # ascending view: strips at the smallest vertex
    assert sum(B.count_shard(g, P.W5, r, 2) for r in range(2)) == exp  # descending: at the largest
    g.close()


@pytest.mark.parametrize("n,p,twins", [
    (64, 0.3, True), (96, 0.5, False), (255, 0.1, True), (257, 0.1, True), (1023, 0.01, True), (1025, 0.01, True),
    (2048, 0.004, True), (2049, 0.004, True), (2079, 0.004, True), (2081, 0.004, True), (16384, 0.0003, True),
    (16385, 0.0003, True)])
def test_hub_neighbourhoods_beside_statistics(ctx, n, p, twins):
    """Beside a statistics form (4-path cone) the 4-wheel is counted from the same rows; above 16,384 neighbours in
    groups of strips."""
    rp, col = hub_over(n, p, twins, n)
    g = B.Graph.from_csr(ctx, rp, col)
    b = B.Batch(ctx)
    path = P.central_patterns(5)[6]
    assert B.Query.from_edges(path).plan()["nbhd"] == 4
    for q in (path, P.W5):
        b.add(g, q)
    assert b.run() == [B.count(g, path, B.SGM, B.OPT_NO_NBHD) if n < 2000 else B.count(g, path),
                       O.count(rp, col, P.W5, apply_root_cap=False)["count"]]
    b.close()
    g.close()


@pytest.mark.parametrize("n,core", [(16500, 40), (16500, 1500), (16500, 2200), (40000, 1500)])
def test_wide_roots_with_a_dense_core(ctx, n, core):
    """A hub over n vertices, `core` of them joined to each other: above a core vertex lie more neighbours than the
    index list holds (1,024), in rows with a list of non-zero words (up to 2,048 of them) and without. The shards count
    on the descending view, with the list kernel."""
    rng = np.random.default_rng(core)
    m = 3 * n
    a, b = np.triu_indices(core, 1)
    us = [np.zeros(n, np.int64), rng.integers(1, n + 1, m), a + 1]
    vs = [np.arange(1, n + 1), rng.integers(1, n + 1, m), b + 1]
    rp, col = synth.to_csr(n + 1, np.concatenate(us), np.concatenate(vs))
    g = B.Graph.from_csr(ctx, rp, col)
    exp = sum(B.count_shard(g, P.W5, r, 2) for r in range(2))
    if core < 100:
        assert exp == O.count(rp, col, P.W5, apply_root_cap=False)["count"]
    assert B.count(g, P.W5) == exp > 0
    bt = B.Batch(ctx)
    path = P.central_patterns(5)[6]
    for q in (P.W5, path):
        bt.add(g, q)
    assert bt.run() == [exp, B.count(g, path)]
    bt.close()
    g.close()
