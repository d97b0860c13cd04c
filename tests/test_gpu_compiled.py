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
