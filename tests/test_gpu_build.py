"""Graph builds from raw inputs: what is refused, and what the build cleans up."""
import numpy as np
import pytest

import beep_b200 as B
from oracle import synth


@pytest.mark.gpu
@pytest.mark.parametrize("extra", [-1, 1, 100000, (1 << 32) - 10])
def test_device_csr_entry_count_mismatch(ctx, extra):
    """An m other than row_ptr[n] is refused before a column entry beyond row_ptr[n] is read or room for m entries
    is made (the largest asks for 17 GB)."""
    import torch

    rp, col = synth.erdos_renyi(500, 0.02, 3)
    d_rp, d_col = (torch.from_numpy(x.astype("int32")).cuda() for x in (rp, col))
    torch.cuda.synchronize()
    m = len(col)
    free = torch.cuda.mem_get_info()[0]
    with pytest.raises(B.BeepError) as e:
        B.Graph.from_device_csr(ctx, 500, extra if extra > 1 << 31 else m + extra, d_rp.data_ptr(), d_col.data_ptr())
    assert e.value.status == 1 and "row_ptr[n] != m" in str(e.value)
    assert free - torch.cuda.mem_get_info()[0] < 1 << 30
    g = B.Graph.from_device_csr(ctx, 500, m, d_rp.data_ptr(), d_col.data_ptr())
    assert g.info()["m"] == m
    g.close()


def raw_edges(kind, n, rng):
    """Edges over ids 0 .. n - 1, the largest used, both directions, unordered, with loops and duplicates."""
    if kind == "loops":
        return np.arange(n, dtype=np.uint32), np.arange(n, dtype=np.uint32)
    u, v = rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)
    last = np.full(3, n - 1)
    u, v = np.concatenate([u, last, last]), np.concatenate([v, last, [0, 0, n // 2]])
    s, d = np.concatenate([u, v, u[: n // 2]]), np.concatenate([v, u, v[: n // 2]])
    order = rng.permutation(len(s))
    return s[order].astype(np.uint32), d[order].astype(np.uint32)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["mixed", "loops"])
@pytest.mark.parametrize("n", [1, 2, 3, 255, 256, 257, 65535, 65536, 65537])
def test_raw_edges(ctx, kind, n):
    """Keys hold two ids of as many bits as the largest needs, and loops share their largest value."""
    src, dst = raw_edges(kind, n, np.random.default_rng(n))
    keep = src != dst
    key = np.unique(src[keep].astype(np.uint64) << 32 | dst[keep])
    g = B.Graph.from_edges(ctx, src, dst)
    rp, col = g.csr()
    assert g.info()["n"] == n and g.info()["m"] == len(key)
    assert np.array_equal(col[: len(key)], (key & 0xFFFFFFFF).astype(np.int32))
    assert np.array_equal(rp, np.searchsorted(key >> 32, np.arange(n + 1)))
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,bad", [(5, 5), (8, 8), (8, 7), (6, 1 << 30)])
def test_unsorted_csr_with_an_id_out_of_range(ctx, n, bad):
    """The sorting path refuses ids of n and more, also those that fit the keys' bits."""
    rp = np.array([0, 3] + [4] * (n - 1), np.int32)
    col = np.array([3, 1, bad, 0], np.int32)  # row 0 unsorted, row 1: {0}
    if bad < n:
        g = B.Graph.from_csr(ctx, rp, col)
        assert g.info()["m"] == 4
        g.close()
        return
    with pytest.raises(B.BeepError) as e:
        B.Graph.from_csr(ctx, rp, col)
    assert e.value.status == 1


@pytest.mark.gpu
def test_round_trip_through_several_chunks(ctx):
    """Columns of 18 MB from and to pageable memory, the last chunk a partial one."""
    rp, col = synth.erdos_renyi(30000, 0.005, 9)
    assert len(col) * 4 > 16 << 20 and len(col) * 4 % (4 << 20)
    g = B.Graph.from_csr(ctx, rp, col)
    got_rp, got_col = g.csr()
    assert np.array_equal(got_rp, rp) and np.array_equal(got_col, col)
    g.close()
