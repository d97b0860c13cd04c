"""Texture editing through the C interface: records that its inputs hold are the
renderer's and are not read, those given as a parameter are."""
import ctypes

import pytest
import torch

from gpu_helpers import Case, small_scene

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("bw", [8, 16])
def test_records_of_the_renderer_are_not_editings(bw):
    """Splats of a third of a pixel under blur, whose alpha comes from the
    filter: records built without blur hold regions that are too small for it.
    With them among the inputs the edit is that of no records; with records
    built for it, given by themselves, too (sums in another order: 1e-5 of a
    row's weights; one row in a hundred on a threshold)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gstex_cuda_gb300 import _lib, cuda as C
    spec = small_scene(n=300, width=48, height=40, seed=7, f=48.0, scale=(0.01, 0.03), chart=(1, 3))
    case = Case(spec)
    b, t = case.binning_cuda(bw), case.t
    L, T, st = _lib.lib(), spec.texture.shape[0], torch.cuda.current_stream().cuda_stream
    g = torch.Generator().manual_seed(1)
    img, alpha = torch.rand(40, 48, 3, generator=g).to(DEV), torch.ones(40, 48, device=DEV)
    lo, hi = torch.zeros(40, 48, device=DEV), torch.full((40, 48), 100.0, device=DEV)
    p = C.ptr
    ri = _lib.RasterInputs()
    ri.num_points, ri.img_width, ri.img_height, ri.block_width = 300, 48, 40, bw
    ri.channels, ri.num_texels = 5, T
    ri.texture_dims, ri.gaussian_ids_sorted, ri.tile_bins = p(t["dims"]), p(b["gaussian_ids_sorted"]), p(b["tile_bins"])
    ri.opacities, ri.means, ri.scales, ri.glob_scale = p(t["opacity"]), p(t["means"]), p(t["scales"]), 1.0
    ri.quats, ri.uv0, ri.umap, ri.vmap, ri.viewmat = p(t["quats"]), p(t["uv0"]), p(t["umap"]), p(t["vmap"]), p(t["viewmat"])
    ri.fx, ri.fy, ri.cx, ri.cy = case.intr
    ri.settings = 1

    def records(settings):
        rr = _lib.RasterInputs.from_buffer_copy(ri)
        rr.channels, rr.num_texels, rr.colors, rr.background, rr.settings = 0, 0, p(t["colors"]), p(t["colors"]), settings
        buf = torch.empty(L.gstex_view_records_bytes(300), dtype=torch.uint8, device=DEV)
        assert L.gstex_view_records(ctypes.byref(rr), p(buf), buf.numel(), st) == 0
        return buf

    def edit(inner, given=None):
        ri.records = p(inner)
        out = torch.full((T, 5), -1.0, device=DEV)
        io = _lib.EditIO(p(img), p(alpha), p(lo), p(hi), T, p(out))
        if given is None:
            assert L.gstex_texture_edit(ctypes.byref(ri), ctypes.byref(io), st) == 0
        else:
            assert L.gstex_texture_edit_records(ctypes.byref(ri), ctypes.byref(io), p(given), st) == 0
        return out

    plain, blurred = records(0), records(1 << 9)
    want = edit(None)
    assert float(want[:, 4].sum()) > 10.0
    for got in (edit(plain), edit(blurred), edit(plain, blurred)):
        bad = (got - want).abs() > 1e-5 * (1 + want.abs())
        assert float(bad.any(1).float().mean()) <= 1e-2
    assert L.gstex_texture_edit_records(ctypes.byref(ri), ctypes.byref(_lib.EditIO()), p(blurred) + 8, st) == 1
