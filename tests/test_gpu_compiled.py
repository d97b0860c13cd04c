"""Calls inside torch.compile (the eager backend: what matters is that the
compiler can read its way through them)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def _require():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch._dynamo.reset()
    yield
    torch._dynamo.reset()


@pytest.mark.parametrize("dynamic", [False, True])
def test_project_points_in_one_graph(dynamic):
    """The torch operations, without a break of the graph."""
    from gstex_cuda_gb300.get_aabb_2d import project_points
    p, vm = torch.randn(64, 3, generator=torch.Generator().manual_seed(0)).to(DEV), torch.eye(4, device=DEV)
    f = lambda x: project_points(x, vm, (400.0, 390.5, 399.5, 300.25))  # noqa: E731
    got = torch.compile(f, backend="eager", fullgraph=True, dynamic=dynamic)(p)
    for x, y in zip(got, f(p.clone().requires_grad_())):
        assert torch.equal(x, y.detach())


def _case():
    from gpu_helpers import Case, small_scene
    case = Case(small_scene(n=120, width=40, height=28, seed=6))
    return case, case.binning_cuda(16), case.t


def test_texture_edit():
    """Around breaks of the graph (the library's calls), the same edit."""
    from gstex_cuda_gb300.texture_edit import texture_edit
    case, b, t = _case()
    g = torch.Generator().manual_seed(1)
    img, alpha = torch.rand(28, 40, 3, generator=g).to(DEV), torch.ones(28, 40, 1, device=DEV)
    lo, hi = torch.zeros(28, 40, device=DEV), torch.full((28, 40), 9.0, device=DEV)

    def edit():
        return texture_edit((120, 1, 5), t["dims"], img, alpha, lo, hi, b["centers"], b["extents"], b["depths"],
                            b["counts"], t["opacity"], t["means"], t["scales"], 1.0, t["quats"], t["uv0"], t["umap"],
                            t["vmap"], t["viewmat"], t["c2w"], *case.intr, 28, 40, 16, 0)

    want = edit()
    # (sums in another order)
    assert float((torch.compile(edit, backend="eager")() - want).abs().max()) <= 1e-5 * float(want.abs().max())


def test_texture_gaussians():
    """The renderer and its gradients likewise."""
    import gstex_cuda_gb300 as G
    case, b, t = _case()
    t["means"].requires_grad_()
    bg = torch.zeros(3, device=DEV)

    def render(means):
        return G.texture_gaussians((120, 1, 3), t["dims"], b["centers"], b["extents"], b["depths"], b["counts"],
                                   t["colors"], t["opacity"], means, t["scales"], 1.0, t["quats"], t["uv0"], t["umap"],
                                   t["vmap"], t["texture"], t["viewmat"], t["c2w"], *case.intr, 28, 40, 16, 1 << 8, bg)

    want, got = render(t["means"]), torch.compile(render, backend="eager")(t["means"])
    for x, y in zip(want, got):
        assert torch.equal(x, y)
    v = [torch.autograd.grad(sum(x.sum() for x in o), t["means"])[0] for o in (want, got)]
    assert float((v[0] - v[1]).abs().max()) <= 1e-5 * float(v[0].abs().max())
