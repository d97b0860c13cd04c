"""Tile counts below 0 (boxes of negative size give them), which make slots
overlap."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def _require():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def test_emission_starts_at_the_first_slot():
    """A sum of counts below 0 is no place in the buffers: nothing is written in
    front of them, and every slot is."""
    from gstex_cuda_gb300 import _lib
    L, n, total = _lib.lib(), 3, 5
    centers, extents = torch.full((n, 2), 24.0, device=DEV), torch.full((n, 2), 10.0, device=DEV)
    depths = torch.ones(n, device=DEV)
    cum = torch.tensor([-4, 1, 5], dtype=torch.int32, device=DEV)  # counts -4, 5, 4
    keys = torch.full((16 + total,), -7, dtype=torch.int64, device=DEV)
    gids = torch.full((16 + total,), -7, dtype=torch.int32, device=DEV)
    assert L.gstex_map_gaussian_to_intersects(n, total, centers.data_ptr(), extents.data_ptr(), depths.data_ptr(),
                                              cum.data_ptr(), 4, 4, 16, 0, keys.data_ptr() + 8 * 16,
                                              gids.data_ptr() + 4 * 16, torch.cuda.current_stream().cuda_stream) == 0
    assert bool((keys[:16] == -7).all()) and bool((gids[:16] == -7).all())
    assert gids[16:].tolist() == [1, 2, 2, 2, 2] and bool((keys[16:] >= 0).all())


@pytest.mark.parametrize("n", [50, 5000])
def test_every_slot_has_an_id(n):
    """As many intersections as the sum of the counts, every one of them a
    Gaussian's, with the tile ranges of the general path.  (Which of two
    Gaussians an overlapping slot goes to is open there as well.)"""
    import gstex_cuda_gb300 as G
    g = torch.Generator().manual_seed(n)
    side, bw = 64, 16
    centers = (bw * (1 + (side - 2) * torch.rand(n, 2, generator=g))).to(DEV)
    extents = torch.full((n, 2), 20.0, device=DEV)
    depths = (1 + torch.rand(n, generator=g)).to(DEV)
    counts = G.get_aabb_2d.get_num_tiles_hit_2d(centers, extents, bw * side, bw * side, bw)
    counts[::7] = -2
    tb = (side, side, 1)
    want, cum = G.utils.compute_cumulative_intersects(counts)
    assert want == int(counts.long().sum())
    spare = torch.full((4 * want,), 0x7FFFFFFF, dtype=torch.int32, device=DEV)  # what an unwritten slot would show
    del spare
    total, gids, bins = G.utils.bin_view(centers, extents, depths, counts, tb, bw)
    assert total == want and int(gids.min()) >= 0 and int(gids.max()) < n
    ids = G.utils.bin_and_sort_gaussians(n, want, centers, extents, depths, cum, tb, bw)
    size = lambda b: (b[:, 1] - b[:, 0]).sum()  # noqa: E731
    assert int(size(bins)) == int(size(ids[4])) == want
