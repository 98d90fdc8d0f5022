"""The row gather at the edges of its items: one row, rows of 16 bytes up to longer than a stage, row counts around the sizes
where an item takes more rows, remainders of an item, more positions than a batch holds. Copies: byte-exact."""

import pytest
import torch

import gpu_util as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,row_bytes", [(1, 16), (31, 48), (2367, 8192), (2368, 8192), (9473, 4096), (9470, 2064), (20001, 5760),
                                         (75777, 512), (75775, 16), (300001, 16), (700, 16400), (1201, 40000), (5, 65536)])
def test_gather_item_edges(native_lib, cuda_device, n, row_bytes):
    gen = torch.Generator(device=cuda_device).manual_seed(n)
    src = max(1, min(n, 5000))
    rows = torch.randint(0, 256, (src, row_bytes), dtype=torch.uint8, device=cuda_device, generator=gen)
    pos = torch.randint(0, src, (n,), dtype=torch.int32, device=cuda_device, generator=gen)
    got, status = G.cuda_gather_rows(rows, pos)
    assert status.tolist() == [0, 0]
    assert torch.equal(got, rows[pos.long()])
    if n > 100:  # a position outside the source: recorded, and the row taken is row 0
        pos[n - 3] = src
        got, status = G.cuda_gather_rows(rows, pos)
        assert status.tolist() == [5, n - 3]
        pos[n - 3] = 0
        assert torch.equal(got, rows[pos.long()])
