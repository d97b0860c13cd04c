"""Quaternions that are not of unit length: their axes are oblique, as in the
reference, which does not normalise them, and so is the region that a splat is
culled by."""
import numpy as np
import pytest
import torch

import oracle
from gpu_helpers import Case, np_, small_scene, upstream

pytestmark = pytest.mark.gpu


def _spec(which):
    spec = small_scene(n=150, width=45, height=31, seed=4, scale=(0.02, 0.6))
    g = torch.Generator().manual_seed(1)
    if which == "lengths":
        spec.quats *= 0.75 + 0.5 * torch.rand(150, 1, generator=g)
    elif which == "components":  # one left out
        spec.quats[torch.arange(150), torch.randint(0, 4, (150,), generator=g)] = 0.0
    elif which == "near one":
        spec.quats *= 1 + 1e-3 * torch.randn(150, 1, generator=g)
    else:
        spec.quats[:] = 0.0
    return spec


@pytest.mark.parametrize("prebuilt", [True, False])
@pytest.mark.parametrize("which", ["lengths", "components", "near one", "none"])
@pytest.mark.parametrize("bw", [8, 16, 5])
def test_no_contributing_pair_is_culled(bw, which, prebuilt):
    """Outputs to 5e-5 of the 64-bit oracle on the same lists (the bar of the
    small scenes, with one value in a thousand on a threshold) and the gradients
    of what does not depend on the axes to 1e-3 of the largest."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gstex_cuda_gb300 as G
    case = Case(_spec(which))
    b = case.binning_cuda(bw)
    gids, bins = b["gaussian_ids_sorted"], b["tile_bins"]
    args = (case.scene_np, case.cam_np, gids.cpu().numpy(), bins.cpu().numpy(), bw, 1 << 8, np.zeros(3))
    ref = oracle.texture_forward(*args, prec="f64")
    ups = upstream(31, 45, 3)
    gref = oracle.texture_backward(*args, ref, *(ups[k] for k in ("img", "depth", "reg", "alpha", "texture", "normal")),
                                   prec="f64")
    G.cuda.PREBUILT_RECORDS = prebuilt
    try:
        out, bg = case.forward_cuda(gids, bins, bw)
        got = case.backward_cuda(out, gids, bins, ups, bw, bg=bg)
    finally:
        G.cuda.PREBUILT_RECORDS = True
    for k in ("img", "texture", "normal", "final_T"):
        err = np.abs(np_(out[k]) - ref[k])
        assert (err > 5e-5).mean() <= 1e-3 and err.max() < 1e-2, (k, float(err.max()), float((err > 5e-5).mean()))
    for k in ("colors", "texture"):
        r = gref[k].reshape(-1)
        assert np.abs(np_(got[k]).reshape(-1) - r).max() <= 1e-3 * np.abs(r).max(), k
