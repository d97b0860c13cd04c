"""Inputs whose element offsets pass 31 bits."""
import pytest
import torch

from gpu_helpers import Case, small_scene, upstream

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def _memory():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("needs 100 GB of free device memory")
    yield
    torch.cuda.empty_cache()


@pytest.mark.parametrize("prebuilt", [True, False])
def test_charts_at_the_end_of_a_large_texture(prebuilt):
    """Float32 texels beyond the 715,827,882th, whose offset in floats passes
    2^31: the same picture as from a small texture, and the same gradients up
    to the order of their sums."""
    import gstex_cuda_gb300 as G
    spec = small_scene(n=80, width=40, height=28, seed=3, chart=(2, 5))
    T0 = spec.texture.shape[0]
    T = 2 ** 31 // 3 + 1 + T0
    case = Case(spec)
    b = case.binning_cuda(8)
    gids, bins = b["gaussian_ids_sorted"], b["tile_bins"]
    ups = upstream(28, 40, 3)
    res = []
    G.cuda.PREBUILT_RECORDS = prebuilt
    try:
        for large in (False, True):
            tex = case.t["texture"]
            if large:
                case.t["dims"][:, 2] += T - T0
                tex = torch.zeros(T, 3, device=DEV)
                tex[T - T0:] = case.t["texture"]
            out, bg = case.forward_cuda(gids, bins, 8, texture=tex)
            g = case.backward_cuda(out, gids, bins, ups, 8, bg=bg, texture=tex)
            res.append((out["texture"], g["texture"][-T0:].clone(), g["means"]))
    finally:
        G.cuda.PREBUILT_RECORDS = True
    assert torch.equal(res[0][0], res[1][0])
    for x, y in zip(res[0][1:], res[1][1:]):
        assert float(x.abs().max()) > 0 and float((x - y).abs().max()) <= 1e-5 * float(x.abs().max())


@pytest.mark.parametrize("used", [0, 1])
def test_sh_of_many_gaussians(used):
    """Colours and their gradients of Gaussians beyond the 715,827,882th equal
    those of a small call on the same rows."""
    import gstex_cuda_gb300 as G
    n, m = 2 ** 31 // 3 + 301, 300
    g = torch.Generator().manual_seed(0)
    dirs, co, up = (torch.randn(*s, generator=g).to(DEV) for s in ((m, 3), (m, 4, 3), (m, 3)))

    def at_the_end(x):
        big = torch.zeros(n, *x.shape[1:], device=DEV)
        big[n - m:] = x
        return big

    far = at_the_end(dirs)
    got = G.cuda.compute_sh_forward(n, 1, used, far, at_the_end(co))[-m:].clone()
    assert torch.equal(got, G.cuda.compute_sh_forward(m, 1, used, dirs, co))
    got = G.cuda.compute_sh_backward(n, 1, used, far, at_the_end(up))[-m:].clone()
    assert torch.equal(got, G.cuda.compute_sh_backward(m, 1, used, dirs, up))


@pytest.mark.parametrize("partial", [False, True])
def test_binning_up_to_the_last_count(partial):
    """524,176 tiles that 4096 Gaussians cover (sorted as one word each), and
    with two more over some of them 2^31 - 1 intersections (sorted as pairs):
    every tile lists the covering Gaussians in depth order, and the compositor
    walks the lists to their ends (the splats are transparent)."""
    import gstex_cuda_gb300 as G
    bw, side, n = 8, 724, 4096
    W = bw * side
    g = torch.Generator().manual_seed(0)
    centers, extents = torch.full((n, 2), W / 2.0), torch.full((n, 2), W / 2.0 - 6)
    depths = 1 + torch.randperm(n, generator=g).float() / n
    rows, strip = 633, 459
    if partial:
        centers = torch.cat([centers, torch.tensor([[W / 2.0, 2528.0], [1836.0, 4.0]])])
        extents = torch.cat([extents, torch.tensor([[W / 2.0 - 6, 2530.0], [1834.0, 2.0]])])
        depths = torch.cat([depths, torch.tensor([3.0, 4.0])])
    N = depths.numel()
    order = torch.argsort(depths[:n]).int().to(DEV)
    centers, extents, depths = centers.to(DEV), extents.to(DEV), depths.to(DEV)
    counts = G.cuda.num_tiles_hit(centers, extents, W, W, bw)
    tb = (side, side, 1)
    total, gids, bins = G.utils.bin_view(centers, extents, depths, counts, tb, bw)
    assert total == side * side * n + (side * rows + strip if partial else 0)
    if partial:
        assert total == 2 ** 31 - 1
    tile = torch.arange(side * side, device=DEV)
    more = torch.stack([tile < side * rows, tile < strip]).long() if partial else torch.zeros(2, 1, device=DEV).long()
    end = (n + more.sum(0)).expand(tile.numel()).cumsum(0)
    start = torch.cat([end.new_zeros(1), end[:-1]])
    assert torch.equal(bins.long(), torch.stack([start, end], 1))
    for at in start.split(8192):
        assert bool((gids[at[:, None] + torch.arange(n, device=DEV)] == order).all())
    if partial:
        assert bool((gids[start[:side * rows] + n] == n).all()) and bool((gids[start[:strip] + n + 1] == n + 1).all())
    z = lambda *s: torch.zeros(*s, device=DEV)  # noqa: E731
    means = torch.cat([z(N, 2), depths[:, None]], 1)
    quats = torch.tensor([1.0, 0.0, 0.0, 0.0], device=DEV).repeat(N, 1)
    dims = torch.tensor([1, 1, 0], dtype=torch.int32, device=DEV).repeat(N, 1)
    eye = torch.eye(4, device=DEV)
    outs = G.cuda.texture_forward(tb, (bw, bw, 1), (W, W, 1), (N, 1, 3), dims, gids, bins, z(N, 3), z(N, 1), means,
                                  z(N, 3) + 1, 1.0, quats, z(N, 1, 2), z(N, 1, 3), z(N, 1, 3), z(1, 3), eye, eye,
                                  float(W), float(W), W / 2.0, W / 2.0, 1 << 8, z(3))
    assert bool((outs[5] == 1).all())


@pytest.mark.parametrize("n", [2, 5000])
def test_as_many_tiles_as_64_bit_keys_take(n):
    """2^30 tiles, which 32-bit keys of a tile and a bit do not hold."""
    import gstex_cuda_gb300 as G
    side, bw = 2 ** 15, 2
    g = torch.Generator().manual_seed(n)
    at = torch.randint(0, side, (n, 2), generator=g)
    depths = 1 + torch.randperm(n, generator=g).float() / n
    tile, order = torch.sort(at[:, 1] * side + at[:, 0])
    centers = (bw * at + 1).float().to(DEV)
    extents = torch.full((n, 2), 0.25, device=DEV)
    counts = torch.ones(n, dtype=torch.int32, device=DEV)
    total, gids, bins = G.utils.bin_view(centers, extents, depths.to(DEV), counts, (side, side, 1), bw)
    assert total == n and torch.equal(gids.cpu().long(), order)  # (no two in one tile)
    assert torch.equal(bins[tile.to(DEV), 0].cpu().long(), torch.arange(n))
    assert int((bins[:, 1] > bins[:, 0]).sum()) == n
