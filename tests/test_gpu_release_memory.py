"""Memory that closed vectors left is kept for the next calls while another vector is alive,
and given back on request; live vectors keep theirs."""
import gc

import numpy as np
import pytest

import pauliprop as pp

pytestmark = pytest.mark.gpu

GIB = 1 << 30


@pytest.mark.parametrize("caps", [[100_000_000], [900_000] * 60])     # blocks of gigabytes; of megabytes
def test_release(caps):
    import torch
    keep = pp.SparsePauliVector(8)
    gc.collect()
    pp.release_memory()
    z = np.arange(1000, dtype=np.uint64).reshape(-1, 1)
    live = pp.SparsePauliVector(64, 1000, 16)
    live.upload(z, z, np.ones(1000), sorted=True)
    before = torch.cuda.mem_get_info()[0]
    vs = [pp.SparsePauliVector(64, c, 16) for c in caps]
    for v in vs:
        v.close()
    assert torch.cuda.mem_get_info()[0] < before - 2 * GIB
    pp.release_memory()
    assert torch.cuda.mem_get_info()[0] > before - (64 << 20)
    assert np.array_equal(live.to_arrays()[0], z)
    live.close()
    keep.close()
