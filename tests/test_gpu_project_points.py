"""project_points in one launch against the torch operations it stands for
(taken whenever something looks at the operations: gradients, forward-mode
tangents, vmap, tracing)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
INTR = (400.0, 390.5, 399.5, 300.25)


@pytest.fixture(scope="module", autouse=True)
def _require():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _inputs(n):
    g = torch.Generator().manual_seed(n)
    q = torch.linalg.qr(torch.randn(3, 3, generator=g))[0]
    vm = torch.eye(4)
    vm[:3, :3] = q
    vm[:3, 3] = torch.randn(3, generator=g)
    return (3 * torch.randn(n, 3, generator=g)).to(DEV), vm.to(DEV)


@pytest.mark.parametrize("n", [0, 1, 2, 31, 255, 256, 257, 5000, 300001])
def test_same_bits_as_the_torch_operations(n):
    from gstex_cuda_gb300.get_aabb_2d import project_points
    p, vm = _inputs(n)
    pix, depth = project_points(p, vm, INTR)
    tp, td = project_points(p.clone().requires_grad_(), vm, INTR)
    assert tp.requires_grad or n == 0
    if n > 16:
        assert torch.equal(depth, td.detach()) and torch.equal(pix, tp.detach())
    else:  # (the library's product of a few rows sums in another order: three roundings of terms below 16)
        assert torch.allclose(depth, td.detach(), rtol=0, atol=3 * 16 * 2.0 ** -24)
    # a strided view of the points, and of the matrix
    wide = torch.zeros(n, 5, device=DEV)
    wide[:, 1:4] = p
    sp, sd = project_points(wide[:, 1:4], vm.T.contiguous().T, INTR)
    assert torch.equal(sd, depth) and torch.equal(sp, pix)


def test_observed_calls_keep_the_torch_operations():
    import torch.autograd.forward_ad as fwAD
    from gstex_cuda_gb300.get_aabb_2d import project_points
    p, vm = _inputs(64)
    pix, depth = project_points(p, vm, INTR)
    t = torch.randn_like(p)
    with fwAD.dual_level():
        _, d = project_points(fwAD.make_dual(p, t), vm, INTR)
        assert torch.allclose(fwAD.unpack_dual(d).tangent, (t @ vm[:3, :3].T)[:, 2], atol=1e-5)
    vd = torch.func.vmap(lambda x: project_points(x, vm, INTR)[1])(torch.stack([p, 2 * p]))
    assert torch.allclose(vd[0], depth, atol=1e-5)
    traced = torch.jit.trace(lambda x: project_points(x, vm, INTR)[1], (p,), check_trace=False)
    assert torch.equal(traced(2 * p), project_points(2 * p, vm, INTR)[1])
    cpu = project_points(p.cpu(), vm.cpu(), INTR)
    assert cpu[1].device.type == "cpu" and torch.allclose(cpu[1], depth.cpu(), atol=1e-5)
    _, dc = project_points(p, vm, INTR, clip=True)
    assert float(dc.min()) == float(torch.tensor(0.01))
