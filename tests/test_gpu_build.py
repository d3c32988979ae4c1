"""Graph builds from raw inputs: what is refused, and what the build cleans up."""
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
