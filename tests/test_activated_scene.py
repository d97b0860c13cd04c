"""The activated scene of raw parameters (no GPU: nothing is launched)."""
import torch

from gstex_cuda_gb300 import batch as B


def test_scenes_over_the_same_means():
    """A raw scene that shares its means with the one before (a trainer that
    replaces its texels, say) has its own texels, charts and colours in the
    activated scene, in the same activated buffers."""
    n, r = 5, object.__new__(B.BatchRenderer)
    r.N, r.dev = n, torch.device("cpu")
    means = torch.zeros(n, 3)

    def raw(scale, means=means):
        return B.RawScene(means=means, raw_scales=torch.zeros(n, 3), raw_quats=torch.zeros(n, 4),
                          mapping=torch.zeros(n, 1, 4), raw_opacity=torch.zeros(n), sh_coeffs=torch.zeros(n, 1, 3),
                          sh_degree=0, texture_dims=torch.zeros(n, 3, dtype=torch.int32), texture=torch.zeros(n, 3),
                          glob_scale=scale)

    first, second = raw(1.0), raw(2.0)
    a = r.activated(first)
    assert r.activated(first) is a and a.texture is first.texture
    b = r.activated(second)
    assert b.texture is second.texture and b.texture_dims is second.texture_dims
    assert b.sh_coeffs is second.sh_coeffs and b.glob_scale == 2.0 and b.means is means
    assert b.scales is a.scales and b.quats is a.quats and b.uv0 is a.uv0 and b.opacity is a.opacity
    assert a.texture is first.texture  # (one that a caller holds stays as it is)
    c = r.activated(raw(1.0, means=torch.ones(n, 3)))
    assert c.scales is not a.scales
