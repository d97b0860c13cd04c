"""gstex_sort_pairs32: stable order at the edges of a sort tile (3072 items), of
the sorts with one launch a pass (152 tiles) and of the digit widths."""
import pytest
import torch

from gstex_cuda_gb300 import batch as B

pytestmark = pytest.mark.gpu

TILE = 3072


def _sort(keys, bits, count=None):
    L, n = B._L(), keys.numel()
    vals = torch.arange(n, dtype=torch.int32, device="cuda")
    ko, vo = torch.full_like(keys, -1), torch.full_like(vals, -1)
    ws = torch.empty(L.gstex_sort32_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    dev = None if count is None else torch.tensor([count], dtype=torch.int64, device="cuda")
    rc = L.gstex_sort_pairs32(n, None if dev is None else dev.data_ptr(), bits, keys.data_ptr(), vals.data_ptr(),
                              ko.data_ptr(), vo.data_ptr(), ws.data_ptr(), ws.numel(),
                              torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return ko, vo


def _check(n, bits, count=None, few=False):
    g = torch.Generator().manual_seed(n + bits)
    top = min(1 << bits, 5) if few else 1 << bits
    keys = (torch.randint(0, top, (n,), generator=g) & 0xFFFFFFFF).to(torch.int64)
    # (two's complement of the unsigned 32-bit key)
    k32 = torch.where(keys >= 1 << 31, keys - (1 << 32), keys).to(torch.int32).cuda()
    ko, vo = _sort(k32, bits, count)
    m = n if count is None else count
    want, order = torch.sort(keys[:m], stable=True)
    assert torch.equal(ko[:m].cpu().to(torch.int64) & 0xFFFFFFFF, want)
    assert torch.equal(vo[:m].cpu().to(torch.int64), order)
    if count is not None:
        assert bool((vo[m:] == -1).all()) and bool((ko[m:] == -1).all())


@pytest.mark.parametrize("n", [2, 33, TILE - 1, TILE, TILE + 1, 151 * TILE + 1, 152 * TILE, 152 * TILE + 1])
@pytest.mark.parametrize("bits", [1, 8, 9, 13, 32])
def test_known_count(n, bits):
    _check(n, bits)


@pytest.mark.parametrize("n", [TILE, 100000, 152 * TILE])
def test_few_values(n):
    _check(n, 32, few=True)


@pytest.mark.parametrize("cap", [2 * TILE, 152 * TILE, 152 * TILE + 1])
@pytest.mark.parametrize("count", [0, 1, TILE, TILE + 1, None])
def test_count_on_device(cap, count):
    _check(cap, 13, cap if count is None else count)
