"""Depth-first binning of one view against the 64-bit keys it replaces: the
same lists and ranges, bit for bit, at the sizes where it changes kernels
(4096 Gaussians or intersections, 1024 slots a warp) and on depths and tile
counts that no projection gives."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module", autouse=True)
def _require():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gstex_cuda_gb300  # noqa: F401


def _inputs(n, w, h, size, seed):
    g = torch.Generator().manual_seed(seed)
    centers = torch.rand(n, 2, generator=g) * torch.tensor([w * 1.2, h * 1.2]) - 0.1 * torch.tensor([w, h])
    extents = size * torch.rand(n, 2, generator=g) + 0.01
    depths = torch.randint(1, max(2, n // 2), (n,), generator=g).float() / 7  # with ties
    return centers.to(DEV), extents.to(DEV), depths.to(DEV)


def _both(centers, extents, depths, counts, w, h, bw):
    import gstex_cuda_gb300 as G
    tb = ((w + bw - 1) // bw, (h + bw - 1) // bw, 1)
    total, cum = G.utils.compute_cumulative_intersects(counts)
    _, _, keys, gids, bins = G.utils.bin_and_sort_gaussians(centers.shape[0], total, centers, extents, depths, cum, tb,
                                                            bw)
    got = G.utils.bin_view(centers, extents, depths, counts, tb, bw)
    assert got[0] == total
    assert torch.equal(got[2], bins)
    listed = int(bins.max())  # (keys of no tile come last, in any order)
    assert torch.equal(got[1][:listed], gids[:listed])
    return total


@pytest.mark.parametrize("n", [1, 2, 33, 1023, 4095, 4096, 4097, 20011])
@pytest.mark.parametrize("w,h,bw,size", [(32, 32, 16, 6.0), (253, 187, 16, 12.0), (640, 400, 8, 3.0), (97, 61, 10, 90.0)])
def test_equals_the_64_bit_sort(n, w, h, bw, size):
    import gstex_cuda_gb300 as G
    c, e, d = _inputs(n, w, h, size, n + w)
    _both(c, e, d, G.get_aabb_2d.get_num_tiles_hit_2d(c, e, h, w, bw), w, h, bw)


@pytest.mark.parametrize("total", [4095, 4096, 4097, 1024 * 9, 1024 * 9 + 1])
def test_number_of_slots(total):
    """One tile, one slot per Gaussian but the last, which takes the rest as zero entries."""
    n = 1500
    c, e, d = _inputs(n, 16, 16, 4.0, total)
    c[:] = 8.0
    counts = torch.ones(n, dtype=torch.int32, device=DEV)
    counts[-1] = total - n + 1
    assert _both(c, e, d, counts, 16, 16, 16) == total


@pytest.mark.parametrize("n", [300, 6000])
@pytest.mark.parametrize("what", ["zero_entries", "negative", "zero_depth", "nan_inf", "none", "truncated", "one_hides_all"])
def test_odd_depths_and_counts(n, what):
    import gstex_cuda_gb300 as G
    c, e, d = _inputs(n, 200, 120, 20.0, 5)
    counts = G.get_aabb_2d.get_num_tiles_hit_2d(c, e, 120, 200, 16)
    if what == "zero_entries":
        e[::7] = 0.0  # emits nothing but keeps its count
    elif what == "negative":
        d[::5] *= -1.0
        d[3] = -0.0
    elif what == "zero_depth":
        d[::9] = 0.0
        e[::7] = 0.0
    elif what == "nan_inf":
        d[::11] = float("nan")
        d[1::11] = float("inf")
        d[2::11] = float("-inf")
    elif what == "none":
        counts[:] = 0
    elif what == "truncated":
        counts = torch.clamp(counts, max=3)
    else:
        counts[:] = 0
        counts[n // 2] = 5000
    if what == "none":
        got = G.utils.bin_view(c, e, d, counts, (13, 8, 1), 16)
        assert got[0] == 0 and got[1].numel() == 0 and int(got[2].abs().sum()) == 0 and tuple(got[2].shape) == (104, 2)
        return
    _both(c, e, d, counts, 200, 120, 16)


@pytest.mark.parametrize("n", [2 ** 18, 2 ** 18 + 1])
@pytest.mark.parametrize("w,h", [(1024, 1024), (1024, 1008)])
def test_key_and_id_in_one_word(n, w, h):
    """18 or 19 bits of id beside 14 or 13 of tile: sorted as one word up to 32."""
    import gstex_cuda_gb300 as G
    c, e, d = _inputs(n, w, h, 12.0, n + h)
    _both(c, e, d, G.get_aabb_2d.get_num_tiles_hit_2d(c, e, h, w, 16), w, h, 16)
