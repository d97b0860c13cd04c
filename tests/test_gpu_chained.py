"""Kernels that are set up while the one before them still runs (chained
launches) read what this pass wrote, not what the last one left in the same
buffers: two scenes in turn through one renderer and one allocator, without a
synchronisation in between."""
import pytest
import torch

from gpu_helpers import small_scene

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PASSES = 40


@pytest.fixture(scope="module", autouse=True)
def _require():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _scenes(n, **kw):
    return [small_scene(n=n, seed=s, chart=(3, 3), **kw) for s in (1, 2)]


@pytest.mark.parametrize("n", [300, 40000])
def test_batch(n):
    from gstex_cuda_gb300 import batch as B
    specs = _scenes(n, width=96, height=80, scale=(0.01, 0.1))
    keys = ("means", "scales", "quats", "opacity", "sh_coeffs", "uv0", "umap", "vmap", "texture_dims", "texture")
    scenes = [B.Scene(**{k: getattr(s, k).to(DEV) for k in keys}, sh_degree=0) for s in specs]
    cam = specs[0].cameras[0]
    cams = [B.Camera(cam.viewmat, cam.fx, cam.fy, cam.cx, cam.cy, cam.width, cam.height) for _ in range(3)]
    r = B.BatchRenderer(cams, n, capacity=1 << 20, block_width=8)
    gen = torch.Generator().manual_seed(1)
    tgt = [torch.rand(r.total_pixels, 3, generator=gen).to(DEV) for _ in range(2)]
    want = []
    for s in scenes:
        torch.cuda.synchronize()
        r.step(s, *tgt)
        torch.cuda.synchronize()
        want.append((r.out["img"].clone(), r.gids_sorted.clone(), r.grads["means"].clone()))
    assert r.check_capacity() and not torch.equal(want[0][0], want[1][0])
    got = []
    for i in range(PASSES):
        r.step(scenes[i & 1], *tgt)
        got.append((r.out["img"].clone(), r.gids_sorted.clone(), r.grads["means"].clone()))
    torch.cuda.synchronize()
    m = int(r.count.item())
    for i, g in enumerate(got):
        w = want[i & 1]
        assert torch.equal(g[0], w[0]), i
        if i & 1:  # (the count is the last pass's)
            assert torch.equal(g[1][:m], w[1][:m]), i
        # float sums in another order: a thousandth of the largest
        assert (g[2] - w[2]).abs().max() <= 1e-3 * w[2].abs().max(), i


@pytest.mark.parametrize("n", [300, 40000])
def test_view(n):
    from gpu_helpers import Case
    cases = [Case(s) for s in _scenes(n, width=96, height=80, scale=(0.01, 0.1))]

    def one(c):
        b = c.binning_cuda(16)
        out, _ = c.forward_cuda(b["gaussian_ids_sorted"], b["tile_bins"], 16, 1 << 8, [0.2, 0.4, 0.1])
        return out["img"], b["gaussian_ids_sorted"], b["tile_bins"]

    want = []
    for c in cases:
        want.append([x.clone() for x in one(c)])
        torch.cuda.synchronize()
    got = [[x.clone() for x in one(cases[i & 1])] for i in range(PASSES)]
    for i, g in enumerate(got):
        assert all(torch.equal(x, y) for x, y in zip(g, want[i & 1])), i
