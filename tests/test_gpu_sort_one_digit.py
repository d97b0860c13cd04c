"""Sorts whose items share a digit in some pass: those passes copy, and the
others see the order that they left."""
import pytest
import torch

from gstex_cuda_gb300 import batch as B, cuda as C

pytestmark = pytest.mark.gpu
TILE = 3072


@pytest.fixture(autouse=True)
def _require():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _keys(n, which):
    g = torch.Generator().manual_seed(n)
    if which == "one":
        return torch.full((n,), 0x5A, dtype=torch.int64)
    if which == "low":
        return torch.randint(0, 5, (n,), generator=g)
    k = 0x33003300 + (torch.randint(0, 256, (n,), generator=g) << 16)  # passes 1, 2 and 4 share a digit
    if which == "one apart":
        k = torch.full((n,), 0x33, dtype=torch.int64)
        k[-1] = 0x32
    return k


@pytest.mark.parametrize("n", [152 * TILE + 1, 500001, 1216 * TILE, 1216 * TILE + 5])
@pytest.mark.parametrize("which", ["one", "low", "middle", "one apart"])
def test_32_and_64_bit_keys(n, which):
    keys = _keys(n, which)
    want, order = torch.sort(keys, stable=True)
    k64, v = keys.cuda(), torch.arange(n, dtype=torch.int32, device="cuda")
    for bits in (45, 64):
        ko, vo = C.sort_pairs(k64, v, bits)
        assert torch.equal(ko.cpu(), want) and torch.equal(vo.cpu().long(), order)
    L, k32 = B._L(), k64.int()
    ws = torch.empty(L.gstex_sort32_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    for count in (None, n, n - 7, TILE, 1, 0):
        ko, vo = torch.full_like(k32, -1), torch.full_like(v, -1)
        dev = None if count is None else torch.tensor([count], dtype=torch.int64, device="cuda")
        assert L.gstex_sort_pairs32(n, None if dev is None else dev.data_ptr(), 32, k32.data_ptr(), v.data_ptr(),
                                    ko.data_ptr(), vo.data_ptr(), ws.data_ptr(), ws.numel(),
                                    torch.cuda.current_stream().cuda_stream) == 0
        m = n if count is None else count
        w, o = torch.sort(keys[:m], stable=True)
        assert torch.equal(ko[:m].cpu().long(), w) and torch.equal(vo[:m].cpu().long(), o)
        assert bool((vo[m:] == -1).all()) and bool((ko[m:] == -1).all())


@pytest.mark.parametrize("n", [152 * TILE + 1, 600001])
def test_one_tile(n):
    """A view of one tile, whose intersections (sorted as one word each) all
    have its key: the Gaussians in depth order."""
    import gstex_cuda_gb300 as G
    depths = 1 + torch.rand(n, generator=torch.Generator().manual_seed(n))
    xy = torch.full((n, 2), 4.0, device="cuda")
    total, gids, bins = G.utils.bin_view(xy, xy / 2, depths.cuda(), torch.ones(n, dtype=torch.int32, device="cuda"),
                                         (1, 1, 1), 8)
    assert total == n and bins.tolist() == [[0, n]]
    assert torch.equal(gids.cpu().long(), torch.sort(depths, stable=True)[1])
