"""The tile kernels' launch knobs in the batch (records not prebuilt, so that
these kernels run): Gaussians a round, resident CTAs and lanes per walk change
how a tile is walked, not what it composites."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
OUTS = ("img", "depth", "reg", "texture", "normal", "final_T", "final_idx", "depth_idx", "reg_s")
GRADS = ("opacity", "means", "scales", "quats", "uv0", "umap", "vmap", "texture", "sh_coeffs")


@pytest.fixture(scope="module")
def scene():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gstex_cuda_gb300 import batch as B, synthetic
    g = torch.Generator().manual_seed(23)
    cams = synthetic.sphere_cameras(g, 3, radius=8.0, resolutions=[(96, 64), (80, 80), (128, 72)])
    spec = synthetic._finish_with_area(g, torch.empty(2500, 3).uniform_(-3, 3, generator=g), 0.01, 0.1, 3, "normal",
                                       cams, 30_000, "multi", {})
    t16 = torch.zeros(spec.texture.shape[0], 4, dtype=torch.bfloat16)
    t16[:, :3] = spec.texture.to(torch.bfloat16)
    s = B.Scene(means=spec.means.to(DEV), scales=spec.scales.to(DEV), quats=spec.quats.to(DEV),
                opacity=spec.opacity.to(DEV), sh_coeffs=spec.sh_coeffs.to(torch.bfloat16).to(DEV), sh_degree=3,
                uv0=spec.uv0.to(DEV), umap=spec.umap.to(DEV), vmap=spec.vmap.to(DEV),
                texture_dims=spec.texture_dims.to(DEV), texture=t16.to(DEV))
    bcams = [B.Camera(c.viewmat, c.fx, c.fy, c.cx, c.cy, c.width, c.height) for c in cams]
    gen = torch.Generator().manual_seed(2)
    P = sum(c.width * c.height for c in cams)
    return s, bcams, spec.num_points, [torch.rand(P, 3, generator=gen).to(DEV) for _ in range(2)]


def _step(scene, records=False, **knobs):
    from gstex_cuda_gb300 import batch as B
    s, cams, n, tgt = scene
    r = B.BatchRenderer(cams, n, texture_dtype=torch.bfloat16, capacity=1 << 20, prebuilt_records=records, **knobs)
    assert r.takes_knobs() is not records
    r.step(s, *tgt)
    return ({k: r.out[k].cpu().numpy() for k in OUTS}, {k: r.grads[k].cpu().numpy() for k in GRADS})


@pytest.mark.parametrize("bw,knobs", [(8, dict(bwd_ctas=10)), (8, dict(bwd_ctas=10, bwd_batch=48)),
                                      (8, dict(bwd_ctas=10, bwd_group=32)), (8, dict(bwd_batch=48, fwd_batch=48)),
                                      (8, dict(fwd_batch=1, bwd_batch=1)), (16, dict(fwd_batch=64, bwd_batch=128)),
                                      (16, dict(bwd_group=4)), (16, dict(bwd_group=16)), (16, dict(bwd_group=32)),
                                      (16, dict(fwd_ppt=2, bwd_ppt=2))])
def test_knobs_do_not_change_results(scene, bw, knobs):
    """Outputs bit for bit, gradients up to the order of the global atomics
    (1e-4 of the largest, as with the block kernels), and both as with the
    block kernels up to rounding."""
    out0, g0 = _step(scene, block_width=bw)
    out1, g1 = _step(scene, block_width=bw, **knobs)
    for k in OUTS:
        if k == "final_idx" or k == "depth_idx" or "fwd_ppt" not in knobs:
            assert np.array_equal(out0[k], out1[k]), k
        else:
            assert np.abs(out0[k] - out1[k]).max() <= 1e-5 * (1 + np.abs(out0[k]).max()), k
    for k in GRADS:
        assert np.abs(g0[k] - g1[k]).max() <= 1e-4 * (np.abs(g0[k]).max() + 1e-12), k
    _, gb = _step(scene, records=True, block_width=bw)
    for k in GRADS:
        assert np.abs(gb[k] - g1[k]).max() <= 1e-3 * (np.abs(g1[k]).max() + 1e-12), k
