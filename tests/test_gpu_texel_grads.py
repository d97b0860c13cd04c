"""Texel gradients of the block compositor where its shortcuts meet values and
pixels that ordinary data do not have: gradients that are not finite, and
pixels on the plane of an edge-on splat."""
import numpy as np
import pytest
import torch

import oracle
from gpu_helpers import Case, np_, small_scene, upstream

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module", autouse=True)
def _require():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _bf16(spec):
    """The scene's texels rounded to bfloat16, and the kernels' padded form of them."""
    tex = spec.texture.to(torch.bfloat16)
    spec.texture = tex.float()
    return torch.cat([tex, torch.zeros(tex.shape[0], 1, dtype=torch.bfloat16)], 1).to(DEV)


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("chart", [(1, 1), (1, 5)])
@pytest.mark.parametrize("bf16", [False, True])
def test_values_that_are_not_finite_stay_in_their_texels(chart, value, bf16):
    """An infinite or undefined gradient of one pixel reaches the texels under
    it and no others: the same elements as with the tile kernels, which add to
    every corner by itself."""
    import gstex_cuda_gb300 as G
    spec = small_scene(n=80, width=40, height=28, seed=3, chart=chart)
    tex = _bf16(spec) if bf16 else None
    case = Case(spec)
    b = case.binning_cuda(8)
    gids, bins = b["gaussian_ids_sorted"], b["tile_bins"]
    ups = upstream(28, 40, 3)
    ups["texture"][14, 20, 1] = value
    bad = []
    for prebuilt in (True, False):
        G.cuda.PREBUILT_RECORDS = prebuilt
        try:
            out, bg = case.forward_cuda(gids, bins, 8, texture=tex)
            g = case.backward_cuda(out, gids, bins, ups, 8, bg=bg, texture=tex)
        finally:
            G.cuda.PREBUILT_RECORDS = True
        bad.append(~torch.isfinite(g["texture"]))
    assert bool(bad[1].any()) and torch.equal(bad[0], bad[1])


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("bw", [8, 16])
def test_pixels_on_the_plane_of_an_edge_on_splat(bw, bf16):
    """A splat seen exactly edge-on (its normal is the x axis, its plane
    x = 2^-19) and a column of pixels whose rays lie in that plane's direction:
    the ray-plane denominator is 0 there, and the reference's clamp of it to
    1e-6 puts the hit at t = 2^-19 / 1e-6 = 1.9.  Its chart has zero uv maps,
    so that all its pixels fall between the same four texels, which makes it a
    coarse one.  Texel gradients against 64 bits: a few roundings a pair and
    sums of at most 17 rows, 1e-4 of the largest."""
    spec = small_scene(n=2, width=33, height=17, seed=1, f=32.0, chart=(2, 3))
    spec.means[:] = torch.tensor([[2.0 ** -19, 0.0, 2.0], [0.1, 0.05, 3.0]])
    spec.quats[:] = torch.tensor([[0.5, 0.5, 0.5, 0.5], [1.0, 0.0, 0.0, 0.0]])
    spec.scales[:, :2] = 0.5
    spec.opacity[:] = 0.6
    spec.umap[:] = spec.vmap[:] = 0.0
    tex = _bf16(spec) if bf16 else None
    case = Case(spec)
    b = case.binning_cuda(bw)
    gids, bins = b["gaussian_ids_sorted"], b["tile_bins"]
    args = (case.scene_np, case.cam_np, gids.cpu().numpy(), bins.cpu().numpy(), bw, 1 << 8, np.zeros(3))
    ref = oracle.texture_forward(*args, prec="f64")
    ups = upstream(17, 33, 3)
    gref = oracle.texture_backward(*args, ref, *(ups[k] for k in ("img", "depth", "reg", "alpha", "texture", "normal")),
                                   prec="f64")["texture"]
    start = int(spec.texture_dims[0, 2])
    own = slice(start, start + int(spec.texture_dims[0, 0] * spec.texture_dims[0, 1]))
    assert np.abs(gref[own]).max() > 1e-2  # (the edge-on splat is seen)
    out, bg = case.forward_cuda(gids, bins, bw, texture=tex)
    got = np_(case.backward_cuda(out, gids, bins, ups, bw, bg=bg, texture=tex)["texture"])[:, :3]
    assert np.abs(got - gref).max() <= 1e-4 * np.abs(gref).max()
