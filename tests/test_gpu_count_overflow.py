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


@pytest.mark.parametrize("total,used", [(5, 5), (64, 64), (65, 64), (2 ** 32 - 1, 64), (2 ** 32, 0), (2 ** 32 + 5, 0)])
def test_batched_emission_beyond_the_capacity(total, used):
    """The batched emission uses as many slots as it has, and none once the
    32-bit offsets of the pairs have wrapped; the overflow is flagged."""
    from gstex_cuda_gb300 import batch as B
    L = B._L()
    cams = [B.Camera(torch.eye(4), 8.0, 8.0, 4.0, 4.0, 8, 8)]
    r = B.BatchRenderer(cams, 2, capacity=64, block_width=8)
    # two pairs of one tile each, the second with the rest of the slots
    r.rects[:] = torch.tensor([[1 << 16, 1 << 16], [1 << 16, 1 << 16]], dtype=torch.int32, device=DEV)
    r.order[:] = torch.tensor([0, 1], dtype=torch.int32, device=DEV)
    low = (total + 2 ** 31) % 2 ** 32 - 2 ** 31  # (the offset's 32 bits)
    r.cum[:] = torch.tensor([1, low], dtype=torch.int64, device=DEV).int()
    r.total[:] = total
    rc = L.gstex_batch_emit_sorted(2, 1, r.views_dev.data_ptr(), r.order.data_ptr(), r.cum.data_ptr(),
                                   r.rects.data_ptr(), r.total.data_ptr(), 64, r.keys.data_ptr(), r.vals.data_ptr(),
                                   r.count.data_ptr(), r.overflow.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and int(r.count) == used and bool(r.overflow) == (total > 64)
