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
