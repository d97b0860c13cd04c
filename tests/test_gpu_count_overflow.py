"""More tile intersections than their integers hold are refused, not wrapped."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module", autouse=True)
def _require():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("n", [4000, 4096, 8192, 3000000])
def test_sums_of_large_tile_counts(n):
    """Counts of 2^20 tiles each (a 16-megapixel picture in 4x4 tiles): the
    4096 counts that one block adds up come to 2^32."""
    import gstex_cuda_gb300 as G
    counts = torch.full((n,), 1 << 20, dtype=torch.int32, device=DEV)
    with pytest.raises(OverflowError, match=str(n << 20)):
        G.utils.compute_cumulative_intersects(counts)
    xy, depths = torch.ones(n, 2, device=DEV), torch.ones(n, device=DEV)
    with pytest.raises(OverflowError, match=str(n << 20)):
        G.utils.bin_view(xy, xy, depths, counts, (1024, 1024, 1), 4)


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 2 ** 21 - 1, 2 ** 21 + 4097])
def test_sums_below_that(n):
    """Every tile of the scan, up to two launches and with three."""
    import gstex_cuda_gb300 as G
    g = torch.Generator().manual_seed(n)
    counts = torch.randint(0, 700, (n,), generator=g, dtype=torch.int32)
    total, cum = G.utils.compute_cumulative_intersects(counts.to(DEV))
    want = counts.long().cumsum(0)
    assert total == int(want[-1]) and torch.equal(cum.cpu().long(), want)
