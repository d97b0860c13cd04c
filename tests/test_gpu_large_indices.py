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
