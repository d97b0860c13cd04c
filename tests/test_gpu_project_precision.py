"""project_points under autocast, with reduced-precision products and of negated
views: the torch operations' results, as with gradients."""
import contextlib

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
INTR = (400.0, 390.5, 399.5, 300.25)


@contextlib.contextmanager
def _precision(mode):
    if mode in (torch.float16, torch.bfloat16):
        with torch.autocast("cuda", dtype=mode):
            yield
        return
    before = torch.get_float32_matmul_precision()
    torch.set_float32_matmul_precision(mode)
    try:
        yield
    finally:
        torch.set_float32_matmul_precision(before)


@pytest.mark.parametrize("mode", [torch.float16, torch.bfloat16, "high", "highest"])
def test_the_same_with_and_without_gradients(mode):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gstex_cuda_gb300.get_aabb_2d import project_points
    g = torch.Generator().manual_seed(0)
    p, vm = (3 * torch.randn(5000, 3, generator=g)).to(DEV), torch.eye(4)
    vm[:3, :3] = torch.linalg.qr(torch.randn(3, 3, generator=g))[0]
    vm[:3, 3] = torch.randn(3, generator=g)
    vm = vm.to(DEV)
    with _precision(mode):
        pix, depth = project_points(p, vm, INTR)
        tp, td = project_points(p.clone().requires_grad_(), vm, INTR)
    assert pix.dtype == tp.dtype and torch.equal(pix, tp.detach()) and torch.equal(depth, td.detach())


@pytest.mark.parametrize("n", [5, 3000])
def test_points_that_are_stored_negated(n):
    """A view that torch negates as it reads it (the imaginary part of a
    conjugate is one): its memory holds the opposite of its values."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gstex_cuda_gb300.get_aabb_2d import project_points
    g = torch.Generator().manual_seed(n)
    p, vm = torch.randn(n, 3, generator=g).to(DEV), torch.eye(4, device=DEV)
    view = torch._neg_view(p)
    assert view.is_neg()
    pix, depth = project_points(view, vm, INTR)
    want, wdepth = project_points(-p, vm, INTR)
    assert torch.allclose(depth, wdepth, rtol=1e-6, atol=1e-6) and torch.allclose(pix, want, rtol=1e-4)
    _, moved = project_points(p, torch._neg_view(-vm), INTR)
    assert torch.allclose(moved, -wdepth, rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("intrinsics", [INTR[:3], INTR[:2], INTR + (1.0,)])
def test_wrong_numbers_of_intrinsics(intrinsics):
    """Refused with the error of the torch operations."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gstex_cuda_gb300.get_aabb_2d import project_points
    p, vm = torch.randn(20, 3, device=DEV), torch.eye(4, device=DEV)
    with pytest.raises(ValueError):
        project_points(p.requires_grad_(), vm, intrinsics)
    with pytest.raises(ValueError):
        project_points(p.detach(), vm, intrinsics)
