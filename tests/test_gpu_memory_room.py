"""A growth that would leave less than 4 GiB of device memory free is refused, also where
several follow each other within the time for which an answer about free memory stands."""
import gc

import pytest

import pauliprop as pp

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def test_growths_in_quick_succession_leave_4_gib():
    import torch
    gc.collect()
    torch.cuda.empty_cache()
    keep = [pp.SparsePauliVector(8)]
    free = torch.cuda.mem_get_info()[0]
    fill = torch.empty(free - 5 * GIB, dtype=torch.uint8, device="cuda")       # 5 GiB stay free
    refused = 0
    try:
        for _ in range(16):
            try:
                keep.append(pp.SparsePauliVector(64, 1_700_000, 16))           # about 100 MiB
            except MemoryError as e:
                assert "4 GiB" in str(e)
                refused += 1
            # (a vector's small workspaces and the 32 MiB pieces memory comes in are not asked about)
            assert torch.cuda.mem_get_info()[0] > 4 * GIB - 256 * (1 << 20)
    finally:
        for v in keep:
            v.close()
        del fill
        torch.cuda.empty_cache()
    assert refused > 0
