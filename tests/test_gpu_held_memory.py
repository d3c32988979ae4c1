"""Device memory that a context keeps after a call: buffers sized by a large input go back with the call."""
import numpy as np
import pytest

import beep_b200 as B
from beep_b200 import patterns as P
from oracle import synth

pytestmark = pytest.mark.gpu


def free_bytes():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_edge_keys_are_given_back(built):
    """20 million raw edges: the keys (two arrays of 8 bytes an edge) are freed; what stays is the uploaded edges (8),
    the sort's scratch (8) and the dropped graph's columns (at most 4). Half of the keys' 320 MB is the slack."""
    n, m = 1 << 16, 20_000_000
    rng = np.random.default_rng(1)
    src, dst = (rng.integers(0, n, m, dtype=np.uint32) for _ in range(2))
    B.Context(0).close()  # what the first context of a process costs is not the build's
    ctx = B.Context(0)
    before = free_bytes()
    g = B.Graph.from_edges(ctx, src, dst)
    assert g.info()["n"] == n and g.info()["m"] == len(np.unique((src.astype(np.uint64) << 16 | dst)[src != dst]))
    g.close()
    held = before - free_bytes()
    ctx.close()
    assert held < (8 + 8 + 4 + 8) * m


def test_tuple_buffer_is_given_back(built):
    rp, col = synth.erdos_renyi(300, 0.1, 2)
    ctx = B.Context(0)
    g = B.Graph.from_csr(ctx, rp, col)
    few, total = B.enumerate_matches(g, P.TRIANGLE, 100000)
    before = free_bytes()
    many, total2 = B.enumerate_matches(g, P.TRIANGLE, 40_000_000)  # room for 480 MB of tuples
    held = before - free_bytes()
    assert total == total2 == len(few) == len(many) and held < 100 << 20
    g.close()
    ctx.close()
