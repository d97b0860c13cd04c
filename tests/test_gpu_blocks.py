"""The block compositor (one warp per 8x4 pixels, one splat list per pixel)
where its lists, masks and shortcuts have edges: lists around its rounds of 32
splats, pictures that cut its blocks, splats whose region is thin, grazing or
near the camera, and pixels that a skipped splat ends.  The oracle is the fp64
restatement; the tile kernels (records built per tile, culled by the screen
box alone) are the second witness of the culling."""
import numpy as np
import pytest
import torch

import oracle
from gpu_helpers import Case, np_, small_scene, upstream

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
GRADS = ("colors", "opacity", "means", "scales", "quats", "uv0", "umap", "vmap", "texture")


@pytest.fixture(scope="module", autouse=True)
def _require():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _check(case, bw, settings=1 << 8, channels=3, flips=0.0):
    """Forward to 5e-5 of the oracle (the bar of the small scenes) but for a
    share of flipped thresholds, gradients to 1e-3 of the largest entry."""
    b = case.binning_cuda(bw)
    gids, bins = b["gaussian_ids_sorted"], b["tile_bins"]
    bg = np.array([0.2, 0.4, 0.1])
    ref = oracle.texture_forward(case.scene_np, case.cam_np, gids.cpu().numpy(), bins.cpu().numpy(), bw, settings, bg,
                                 prec="f64")
    out, bgt = case.forward_cuda(gids, bins, bw, settings, bg)
    for k in ("img", "texture", "normal", "final_T"):
        if np.size(ref[k]):
            err = np.abs(np_(out[k]) - ref[k])
            assert (err > 5e-5).mean() <= flips and err.max() < 1e-2, (k, float(err.max()), float((err > 5e-5).mean()))
    ups = upstream(case.cam.height, case.cam.width, channels)
    gref = oracle.texture_backward(case.scene_np, case.cam_np, gids.cpu().numpy(), bins.cpu().numpy(), bw, settings,
                                   bg, ref, *(ups[k] for k in ("img", "depth", "reg", "alpha", "texture", "normal")),
                                   prec="f64")
    g = case.backward_cuda(out, gids, bins, ups, bw, settings, bgt)
    for k in GRADS:
        r = gref[k].reshape(-1)
        if r.size:
            err = np.abs(np_(g[k]).reshape(-1) - r).max() / (np.abs(r).max() + 1e-12)
            assert err < 1e-3, (k, err)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 97])
@pytest.mark.parametrize("bw", [8, 16])
def test_list_lengths(n, bw):
    """Every splat covers the picture faintly, so the lists of all pixels have
    n entries and none saturates."""
    spec = small_scene(n=n, width=21, height=18, seed=n, scale=(0.6, 2.0), z=(1.0, 2.0))
    spec.opacity[:] = 0.01 + 0.02 * spec.opacity
    _check(Case(spec), bw)


@pytest.mark.parametrize("w,h", [(1, 1), (8, 4), (9, 5), (7, 33), (40, 3)])
def test_cut_blocks(w, h):
    spec = small_scene(n=120, width=w, height=h, seed=w, f=24.0, scale=(0.05, 0.4))
    _check(Case(spec), 8)
    _check(Case(spec), 16)


@pytest.mark.parametrize("settings", [0, 1 << 8, (1 << 8) | (1 << 2), (1 << 8) | (1 << 9), (1 << 8) | (1 << 10),
                                      (1 << 8) | (1 << 9) | (1 << 10) | (1 << 15)])
@pytest.mark.parametrize("channels", [0, 3])
def test_settings(settings, channels):
    spec = small_scene(n=150, width=40, height=28, seed=4, channels=channels)
    _check(Case(spec), 8, settings, channels, flips=1e-3)


def _tile_path(case, bw, settings=1 << 8):
    import gstex_cuda_gb300 as G
    b = case.binning_cuda(bw)
    outs = []
    for prebuilt in (True, False):
        G.cuda.PREBUILT_RECORDS = prebuilt
        try:
            outs.append(case.forward_cuda(b["gaussian_ids_sorted"], b["tile_bins"], bw, settings)[0])
        finally:
            G.cuda.PREBUILT_RECORDS = True
    return outs


@pytest.mark.parametrize("which", ["thin", "grazing", "near", "tiny", "faint", "large"])
def test_culled_regions_match_the_box_walk(which):
    """No (splat, pixel) pair that contributes is culled: the same last
    contributor and outputs as the tile kernels, which test the box only.
    (Both evaluate a pair with the same operations, but derive the records in
    different kernels: 1e-5 covers the rounding, and one pixel in a thousand
    may sit on a threshold.)"""
    spec = small_scene(n=3000, width=200, height=144, seed=8, scale=(0.01, 0.2))
    n = spec.num_points
    g = torch.Generator().manual_seed(3)
    if which == "thin":
        spec.scales[:, 0] *= 20.0
        spec.scales[:, 1] *= 0.02
    elif which == "grazing":  # normals at right angles to the viewing ray, but for a little
        d = spec.means / spec.means.norm(dim=1, keepdim=True)
        a = torch.linalg.cross(d, torch.randn(n, 3, generator=g))
        nrm = a / a.norm(dim=1, keepdim=True) + d * 0.04 * torch.randn(n, 1, generator=g)
        nrm = nrm / nrm.norm(dim=1, keepdim=True)
        z = torch.tensor([0.0, 0.0, 1.0]).expand(n, 3)
        axis = torch.linalg.cross(z, nrm)
        q = torch.cat([1 + (z * nrm).sum(1, keepdim=True), axis], 1)
        spec.quats[:] = q / q.norm(dim=1, keepdim=True)
    elif which == "near":
        spec.means[:, 2] = 0.05 + 0.5 * torch.rand(n, generator=g)
        spec.means[:, :2] *= 0.2
    elif which == "tiny":
        spec.scales *= 0.02
    elif which == "faint":
        spec.opacity[:] = (1.0 / 255) * (0.98 + 0.1 * spec.opacity)
    else:
        spec.scales *= 20.0
        spec.opacity *= 0.05
    for bw in (8, 16):
        new, old = _tile_path(Case(spec), bw)
        same = (new["final_idx"] == old["final_idx"]).float().mean()
        assert float(same) >= 0.999, float(same)
        for k in ("img", "texture", "normal", "final_T", "depth"):
            err = (new[k] - old[k]).abs() / (1 + old[k].abs())
            assert float((err > 1e-5).float().mean()) <= 1e-3, (k, float(err.max()))


def test_skipped_splat_ends_a_pixel():
    """After three splats of opacity 1 - (1.002e-4)^(1/3) that fill the picture
    T is 1.002e-4.  A later splat with alpha in (0.002, 1/255) is skipped, but
    it ends the pixel (texture.cu:213-221) before the last, strong splat is
    reached; where its alpha is below 0.002 the last splat ends the pixel.  The
    last contributor and the sums are the same either way, so the check is
    against the oracle with a faint fourth contributor: alpha just above 1/255
    leaves T at 0.9983e-4 and would end the pixel, too.  A weaker start (T =
    1.008e-4) lets the faint splats contribute in turn."""
    for t0 in (1.002e-4, 1.006e-4, 1.0095e-4):
        n = 60
        spec = small_scene(n=n, width=32, height=32, seed=2, scale=(0.05, 0.15), z=(2.5, 3.5))
        spec.means[:3, :2] = 0.0
        spec.means[:3, 2] = torch.tensor([1.0, 1.1, 1.2])
        spec.quats[:3] = torch.tensor([1.0, 0.0, 0.0, 0.0])
        spec.scales[:3, :2] = 500.0
        spec.opacity[:3] = 1.0 - t0 ** (1.0 / 3.0)
        spec.opacity[3:] = torch.linspace(0.001, 0.006, n - 3)[:, None]
        spec.umap[:3] = spec.vmap[:3] = 0.0
        case = Case(spec)
        b = case.binning_cuda(8)
        gids, bins = b["gaussian_ids_sorted"], b["tile_bins"]
        out, _ = case.forward_cuda(gids, bins, 8)
        ref = oracle.texture_forward(case.scene_np, case.cam_np, gids.cpu().numpy(), bins.cpu().numpy(), 8, 1 << 8,
                                     np.zeros(3), prec="f64")
        # the tile kernels walk every splat in order
        new, old = _tile_path(case, 8)
        assert float((new["final_idx"] == old["final_idx"]).float().mean()) >= 0.99
        np.testing.assert_allclose(np_(out["final_T"]), ref["final_T"], atol=5e-7)
        np.testing.assert_allclose(np_(out["img"]), ref["img"], atol=2e-5)


@pytest.mark.parametrize("hooks", [False, True])
def test_backward_of_some_outputs_and_again(hooks):
    """Outputs without a gradient count as zero gradients, a second backward
    over a retained graph gives the same, and saved tensors may come back
    through hooks (the splat records are among them)."""
    import contextlib

    import gstex_cuda_gb300 as G
    spec = small_scene(n=120, width=40, height=28, seed=6)
    case = Case(spec)
    t = case.t
    names = ("colors", "opacity", "means", "scales", "quats", "uv0", "umap", "vmap", "texture")
    for k in names:
        t[k].requires_grad_()
    b = case.binning_cuda(16)
    ctx = torch.autograd.graph.save_on_cpu() if hooks else contextlib.nullcontext()
    with ctx:
        outs = G.texture_gaussians((spec.num_points, 1, 3), t["dims"], b["centers"], b["extents"], b["depths"],
                                   b["counts"], t["colors"], t["opacity"], t["means"], t["scales"], 1.0, t["quats"],
                                   t["uv0"], t["umap"], t["vmap"], t["texture"], t["viewmat"], t["c2w"], *case.intr,
                                   28, 40, 16, 1 << 8, torch.zeros(3, device=DEV))
    g = torch.Generator().manual_seed(0)
    ups = [torch.randn(o.shape, generator=g).to(DEV) for o in outs]
    ins = [t[k] for k in names]
    full = [u if k in (0, 4) else torch.zeros_like(u) for k, u in enumerate(ups)]
    ref = torch.autograd.grad(outs, ins, full, retain_graph=True)
    for _ in range(2):
        got = torch.autograd.grad((outs[0], outs[4]), ins, (ups[0], ups[4]), retain_graph=True)
        for k, x, y in zip(names, got, ref):
            # (sums in another order: 1e-5 of the largest entry)
            assert float((x - y).abs().max()) <= 1e-5 * float(y.abs().max()) + 1e-12, k


@pytest.mark.parametrize("bw", [8, 16])
@pytest.mark.parametrize("settings", [0, 1])
def test_edit_matches_the_tile_kernel(bw, settings):
    """Texture editing by blocks against one CTA per tile: sums in another
    order (1e-5 of a row's weights), one texel row in a thousand on a
    threshold; and an infinite edited pixel spoils the same texels."""
    import gstex_cuda_gb300 as G
    spec = small_scene(n=400, width=61, height=43, seed=12, chart=(1, 5))
    case = Case(spec)
    b, t, cam = case.binning_cuda(bw), case.t, case.cam
    T = spec.texture.shape[0]
    g = torch.Generator().manual_seed(1)
    img, alpha = torch.rand(43, 61, 3, generator=g), (torch.rand(43, 61, generator=g) > 0.3).float()
    lo, hi = 3.0 - torch.rand(43, 61, generator=g), 3.0 + torch.rand(43, 61, generator=g)
    img[20, 30, 1] = float("inf")
    alpha[20, 30] = 1.0
    outs = []
    for prebuilt in (True, False):
        G.cuda.PREBUILT_RECORDS = prebuilt
        try:
            outs.append(G.cuda.texture_edit(b["tile_bounds"], (bw, bw, 1), (61, 43, 1), (400, 1, 5), T, t["dims"],
                                            *(x.to(DEV) for x in (img, alpha, lo, hi)), b["gaussian_ids_sorted"],
                                            b["tile_bins"], t["opacity"], t["means"], t["scales"], 1.0, t["quats"],
                                            t["uv0"], t["umap"], t["vmap"], t["viewmat"], t["c2w"], *case.intr,
                                            settings, None))
        finally:
            G.cuda.PREBUILT_RECORDS = True
    new, old = outs
    assert torch.equal(torch.isfinite(new), torch.isfinite(old)) and not torch.isfinite(old).all()
    fine = torch.isfinite(old)
    bad = ((new - old).abs() > 1e-5 * (1 + old.abs())) & fine
    assert float(bad.any(1).float().mean()) <= 1e-3


@pytest.mark.parametrize("chart", [(1, 1), (1, 5), (2, 16)])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_texel_gradient_words(chart, offset):
    """Gradients of float32 texels leave as 16-byte words: charts that start at
    every place within one, a buffer that does too, and its ends, beyond which
    nothing is touched (-0 + 0 would turn the guards into +0)."""
    from gstex_cuda_gb300 import batch as B
    spec = small_scene(n=80, width=40, height=28, seed=offset, chart=chart)
    _check(Case(spec), 8)
    cam = spec.cameras[0]
    scene = B.Scene(**{k: getattr(spec, k).to(DEV) for k in ("means", "scales", "quats", "opacity", "sh_coeffs", "uv0",
                                                             "umap", "vmap", "texture_dims", "texture")}, sh_degree=0)
    r = B.BatchRenderer([B.Camera(cam.viewmat, cam.fx, cam.fy, cam.cx, cam.cy, cam.width, cam.height)],
                        spec.num_points, capacity=1 << 14, block_width=8)
    gen = torch.Generator().manual_seed(1)
    tgt = [torch.rand(r.total_pixels, 3, generator=gen).to(DEV) for _ in range(2)]
    r.step(scene, *tgt)
    want = r.grads["texture"].clone()
    n = want.numel()
    buf = torch.full((n + 16,), -0.0, device=DEV)
    r.grads["texture"] = buf[4 + offset:4 + offset + n].view(-1, 3)
    r.step(scene, *tgt)
    # the sums' order differs between two runs: 80 splats' pairs over a few pixels each
    assert (r.grads["texture"] - want).abs().max() <= 1e-5 * want.abs().max()
    guard = torch.cat([buf[:4 + offset], buf[4 + offset + n:]])
    assert bool(torch.signbit(guard).all()) and bool((guard == 0).all())
