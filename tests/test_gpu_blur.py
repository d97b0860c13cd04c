"""Gradients with the screen-space blur: a pair takes the larger of the
splat's own falloff and the blur filter's, and only pairs of the second kind
have a gradient of the filter's centre."""
import numpy as np
import pytest
import torch

import oracle
from gpu_helpers import Case, np_, small_scene, upstream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [0.5, 10.0, 150.0])
@pytest.mark.parametrize("bw", [8, 16])
def test_mean_gradient_of_small_and_large_splats(sigma, bw):
    """One splat of `sigma` pixels that faces the camera, random gradients of
    the picture.  A splat of half a pixel takes the filter everywhere, one of
    10 or 150 pixels nowhere.  Bound: single-precision rounding
    of a few operations a pixel and of the sums, against terms that partly
    cancel; 1e-4 of the largest component leaves a factor of ten."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    W, H, f = 96, 88, 96.0
    spec = small_scene(n=1, width=W, height=H, seed=2, f=f, chart=(1, 1))
    spec.means[:] = torch.tensor([[0.013, -0.021, 2.0]])
    spec.quats[:] = torch.tensor([[1.0, 0.0, 0.0, 0.0]])
    spec.scales[:, :2] = sigma * 2.0 / f
    spec.opacity[:] = 0.7
    settings = (1 << 8) | (1 << 9)
    case = Case(spec)
    b = case.binning_cuda(bw)
    gids, bins = b["gaussian_ids_sorted"], b["tile_bins"]
    args = (case.scene_np, case.cam_np, gids.cpu().numpy(), bins.cpu().numpy(), bw, settings, np.zeros(3))
    ref = oracle.texture_forward(*args, prec="f64")
    ups = upstream(H, W, 3)
    for k in ("depth", "reg", "texture", "normal"):
        ups[k] *= 0.0
    gref = oracle.texture_backward(*args, ref, *(ups[k] for k in ("img", "depth", "reg", "alpha", "texture", "normal")),
                                   prec="f64")["means"]
    out, bg = case.forward_cuda(gids, bins, bw, settings)
    got = np_(case.backward_cuda(out, gids, bins, ups, bw, settings, bg)["means"])
    err = np.abs(got - gref).max() / np.abs(gref).max()
    assert err <= 1e-4, err
