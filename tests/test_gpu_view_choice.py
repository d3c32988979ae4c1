"""Which peeled and ordered view of a graph each pair of a call is counted on: a view that a call has built is cached,
so asking for it afterwards launches nothing."""
import numpy as np
import pytest

import beep_b200 as B
from beep_b200 import patterns as P
from oracle import synth

pytestmark = pytest.mark.gpu


def built(ctx, g, min_qdeg, asc):
    before = ctx.kernel_launches()
    g.view(min_qdeg, asc)
    return ctx.kernel_launches() == before


@pytest.fixture()
def graph(ctx):
    rp, col = synth.chung_lu(3000, 12.0, 2.1, 8)
    g = B.Graph.from_csr(ctx, rp, col)
    yield g
    g.close()


def run(ctx, g, queries):
    b = B.Batch(ctx)
    for q in queries:
        b.add(g, q)
    counts = b.run(B.OPT_NO_GRAPH)
    b.close()
    return counts


def test_wheel_alone(ctx, graph):
    B.count(graph, P.W5)
    assert built(ctx, graph, 3, True)


def test_wheel_beside_triangle_forms(ctx, graph):
    """The 4-wheel's view is peeled for it (threshold 3), whatever the triangle forms need."""
    counts = run(ctx, graph, [P.TAILED_TRIANGLE, P.W5])
    assert built(ctx, graph, 3, True)
    assert counts == [B.count(graph, q, B.SGM, B.OPT_NO_NBHD) for q in (P.TAILED_TRIANGLE, P.W5)]


@pytest.mark.parametrize("degree,asc", [(16385, True), (262144, True), (262145, False)])
def test_wheel_on_wide_roots(ctx, degree, asc):
    """Above 262,144 neighbours the list kernel takes over, and with it the plan's descending order."""
    rng = np.random.default_rng(3)
    u, v = rng.integers(1, degree + 1, (2, degree // 8))
    rp, col = synth.to_csr(degree + 1, np.concatenate([np.zeros(degree, np.int64), u]),
                           np.concatenate([np.arange(1, degree + 1), v]))
    g = B.Graph.from_csr(ctx, rp, col)
    run(ctx, g, [P.W5])
    assert built(ctx, g, 3, asc)
    g.close()


def test_statistics_beside_triangle_forms(ctx, graph):
    """The statistics forms' view is peeled for them alone (thresholds 2 and 3), whatever the triangle forms need."""
    five = P.central_patterns(5)
    queries = [P.TAILED_TRIANGLE, five[9], five[7], P.W5]
    counts = run(ctx, graph, queries)
    assert built(ctx, graph, 2, True)
    assert counts == [B.count(graph, q, B.SGM, B.OPT_NO_NBHD) for q in queries]


@pytest.mark.parametrize("shared", [P.TAILED_TRIANGLE, P.central_patterns(5)[6]], ids=["triangle_form", "statistics_form"])
def test_clique_views_of_a_graph_that_comes_back(ctx, graph, shared):
    """A first call builds one view for all its patterns; a graph that keeps being counted gets the cliques' own."""
    queries = [shared, P.K4, P.K5]
    before = ctx.kernel_launches()
    first = run(ctx, graph, queries)
    after = ctx.kernel_launches()
    assert run(ctx, graph, queries) == first
    again = ctx.kernel_launches()
    assert after - before > again - after  # a view is built in the first call ...
    for _ in range(15):
        assert run(ctx, graph, queries) == first
    assert built(ctx, graph, 3, True) and built(ctx, graph, 4, True)
    assert first == [B.count(graph, q, B.SGM, B.OPT_NO_NBHD) for q in queries]


def test_clique_views_stay_unbuilt_at_first(ctx, graph):
    for _ in range(3):
        run(ctx, graph, [P.TAILED_TRIANGLE, P.K4])
    assert built(ctx, graph, 1, True) and not built(ctx, graph, 3, True)
