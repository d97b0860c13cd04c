"""Workspace sizes of the sorts over the whole range of their counts (no GPU:
nothing is launched)."""
from gstex_cuda_gb300 import batch as B

LAST = 2 ** 31 - 1
TILE, MAX_BLOCKS, ROW = 3072, 1216, 256 * 4  # items a block takes at a time, blocks, bytes of one block's counts


def test_workspace_at_the_largest_count():
    """The scratch of 2^31 - 1 items holds the second buffers and the counts of
    as many blocks as the launch has, which are nearly all of MAX_BLOCKS."""
    L = B._L()
    for n in (LAST, LAST - TILE, LAST - 1500000):
        tiles = -(-n // TILE)
        blocks = -(-tiles // -(-tiles // MAX_BLOCKS))
        assert blocks > 1200
        assert L.gstex_sort32_workspace_bytes(n) >= 8 * n + blocks * ROW
        assert L.gstex_sort_workspace_bytes(n) >= 12 * n + blocks * ROW
        assert L.gstex_view_bins_workspace_bytes(n) >= 20 * n + blocks * ROW
