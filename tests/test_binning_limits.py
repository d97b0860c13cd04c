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


def test_workspaces_grow_with_the_count():
    """A workspace sized for n items is enough for any fewer: its size never
    falls, also where the launches change (152 sort tiles of 32-bit keys, 1216
    and multiples of it)."""
    L = B._L()
    edges = [TILE * t for t in (1, 151, 152, 153, 156, 304, 608, MAX_BLOCKS, 2 * MAX_BLOCKS, 100 * MAX_BLOCKS)]
    counts = sorted({1, 2, 4096, 4097, 100000, 417000, 466500, LAST} | {max(1, e + d) for e in edges for d in (-1, 0, 1)})
    for size in (L.gstex_sort32_workspace_bytes, L.gstex_sort_workspace_bytes, L.gstex_view_order_workspace_bytes,
                 L.gstex_view_bins_workspace_bytes, L.gstex_batch_tile_order_workspace_bytes):
        got = [size(n) for n in counts]
        assert got == sorted(got), size.__name__
        for n, b in zip(counts, got):
            assert size(max(1, n - n // 9)) <= b
