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
