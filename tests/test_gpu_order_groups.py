"""The forward's queue order when order_group changes between captures."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _renderer():
    from gpu_helpers import small_scene
    from gstex_cuda_gb300 import batch as B
    spec = small_scene(n=300, width=120, height=88, seed=4)
    cam = spec.cameras[0]
    scene = B.Scene(**{k: getattr(spec, k).to(DEV) for k in ("means", "scales", "quats", "opacity", "sh_coeffs", "uv0",
                                                             "umap", "vmap", "texture_dims", "texture")}, sh_degree=0)
    r = B.BatchRenderer([B.Camera(cam.viewmat, cam.fx, cam.fy, cam.cx, cam.cy, cam.width, cam.height)] * 2,
                        spec.num_points, capacity=1 << 16, block_width=8)
    g = torch.Generator().manual_seed(1)
    return r, scene, [torch.rand(r.total_pixels, 3, generator=g).to(DEV) for _ in range(2)]


def _order(r, scene, tgt, group):
    r.order_group = group
    r.step(scene, *tgt)
    return r.tile_order.clone()


def test_a_captured_order_outlives_a_change():
    """A graph keeps reading the groups of the order_group it was captured
    with; a later one leaves them where they are."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r, scene, tgt = _renderer()
    want = _order(r, scene, tgt, 4)
    groups = r._tile_groups()
    at, rows = groups.data_ptr(), groups.clone()
    r.capture(scene, *tgt)
    assert not torch.equal(_order(r, scene, tgt, 2), want)
    del groups
    spare = [torch.full_like(rows, -1) for _ in range(64)]  # would take a freed buffer's place
    r.order_group = 4
    assert r._tile_groups().data_ptr() == at and torch.equal(r._tile_groups(), rows)
    r.replay()
    assert torch.equal(r.tile_order, want)
    del spare


@pytest.mark.parametrize("group", [1, 3, 64])
def test_a_change_within_a_capture(group):
    """An order_group that is new to the renderer can be captured without a
    step before it."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r, scene, tgt = _renderer()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        r.step(scene, *tgt)
    torch.cuda.current_stream().wait_stream(side)
    r.order_group = group
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        r.step(scene, *tgt)
    g.replay()
    got = r.tile_order.clone()
    assert torch.equal(got, _order(r, scene, tgt, group))
