"""The allocation-free entry point through the tier kernels: every central
pattern equals the walk's count (the oracle's for the 4-wheel and the cliques,
which have no walk here) on graphs with empty rows, domains of every tier and
more vertices than the scratch array can classify."""
import numpy as np
import pytest

import beep_b200 as B
from beep_b200 import patterns as P
from oracle import pyoracle as O
from oracle import synth

pytestmark = pytest.mark.gpu


def device_count(rp, col, q, mode=B.SGM):
    import torch

    drp = torch.from_numpy(np.ascontiguousarray(rp, np.int32)).cuda()
    dcol = torch.from_numpy(np.ascontiguousarray(col, np.int32)).cuda()
    torch.cuda.synchronize()
    return B.count_noalloc(0, len(rp) - 1, len(col), drp.data_ptr(), dcol.data_ptr(), q, mode)


def graphs():
    rng = np.random.default_rng(1)
    yield "er", synth.erdos_renyi(900, 0.03, 5)
    yield "power", synth.chung_lu(3000, 14.0, 2.1, 7)
    # ids spread out: most rows are empty, hubs have the lowest ids
    rp, col = synth.chung_lu(800, 16.0, 2.1, 9)
    src = np.repeat(np.arange(800), np.diff(rp)) * 97
    yield "gaps", synth.to_csr(80000, src, col.astype(np.int64) * 97)
    n = 1500
    yield "hub", synth.to_csr(n + 1, np.concatenate([np.zeros(n, np.int64), rng.integers(1, n + 1, 6000)]),
                              np.concatenate([np.arange(1, n + 1), rng.integers(1, n + 1, 6000)]))


@pytest.mark.parametrize("name,csr", list(graphs()), ids=lambda x: x if isinstance(x, str) else "")
def test_central_patterns(ctx, name, csr):
    rp, col = csr
    g = B.Graph.from_csr(ctx, rp, col)
    k6 = P._undirected([(a, b) for b in range(6) for a in range(b)])
    for q in [P.TRIANGLE, P.WEDGE, k6] + P.central_patterns(4) + P.central_patterns(5):
        if q == P.W5 or B.Query.from_edges(q).plan()["restricted"]:
            exp = O.count(rp, col, q, apply_root_cap=False)["count"]
        else:
            exp = B.count(g, q, B.SGM, B.OPT_NO_NBHD)
        assert device_count(rp, col, q) == exp, q
    g.close()


def test_more_vertices_than_the_scratch_classifies(ctx):
    """4.2 million vertices: the block-per-vertex kernel, as before."""
    rp, col = synth.erdos_renyi(2000, 0.01, 3)
    n = 4_200_000
    big = np.concatenate([rp, np.full(n - 2000, rp[-1], rp.dtype)])
    for q in (P.TRIANGLE, P.K4, P.W5):
        assert device_count(big, col, q) == O.count(rp, col, q, apply_root_cap=False)["count"]
