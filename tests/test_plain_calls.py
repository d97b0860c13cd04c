"""Which calls a kernel launch may stand for (no GPU: the tensors' places are
stood in for)."""
from types import SimpleNamespace

import pytest
import torch

from gstex_cuda_gb300 import _lib


@pytest.mark.parametrize("places,current,want", [((0,), 0, True), ((1,), 0, False), ((1, 1), 1, True),
                                                 ((0, 1), 0, False), ((0, 1), 1, False)])
def test_launches_go_to_the_current_device(places, current, want, monkeypatch):
    """A launch goes to the current device, so tensors of another one keep the
    torch operations, which go to theirs."""
    monkeypatch.setattr(torch.cuda, "current_device", lambda: current)
    assert _lib.on_current_device(*(SimpleNamespace(get_device=lambda p=p: p) for p in places)) is want


def test_projection_asks_for_the_current_device(monkeypatch):
    """project_points asks before it launches: with CPU tensors that pass for
    CUDA ones of another device it takes the torch operations."""
    from gstex_cuda_gb300 import get_aabb_2d as A

    class Elsewhere:
        """The parts of a tensor that plain_cuda_f32 reads."""
        is_cuda, dtype, requires_grad, layout = True, torch.float32, False, torch.strided

        def is_neg(self):
            return False

        def get_device(self):
            return 1

    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch, "Tensor", Elsewhere)
    assert not _lib.plain_cuda_f32(Elsewhere(), Elsewhere())
    monkeypatch.undo()
    seen = []
    monkeypatch.setattr(_lib, "plain_cuda_f32", lambda *t: seen.append(len(t)))
    pix, depth = A.project_points(torch.ones(3, 3), torch.eye(4), (1.0, 1.0, 0.0, 0.0))
    assert seen == [2] and depth.tolist() == [1.0, 1.0, 1.0]


def test_products_in_another_type(monkeypatch):
    """Autocast and torch's reduced-precision products change the torch
    operations' results; a launch, which computes in float32, does not stand
    for them then."""
    assert _lib.full_f32_products()
    with monkeypatch.context() as m:
        m.setattr(torch, "is_autocast_enabled", lambda device: device == "cuda")
        assert not _lib.full_f32_products()
    for precision in ("high", "medium"):
        monkeypatch.setattr(torch, "get_float32_matmul_precision", lambda: precision)
        assert not _lib.full_f32_products()

    def mixed():
        raise RuntimeError("set through both interfaces")

    monkeypatch.setattr(torch, "get_float32_matmul_precision", mixed)
    assert not _lib.full_f32_products()


@pytest.mark.parametrize("where,name", [(torch._C, "_functorch"), (torch._C, "_get_tracing_state"),
                                        (torch._C, "_len_torch_dispatch_stack"),
                                        (torch._C, "_len_torch_function_stack"),
                                        (torch.autograd.forward_ad, "_current_level")])
def test_a_torch_without_one_of_its_private_names(where, name, monkeypatch):
    """Names that torch does not promise: without one the torch operations are
    kept."""
    assert _lib.unobserved()
    monkeypatch.delattr(where, name)
    assert not _lib.unobserved()


def test_streams_without_the_raw_lookup(monkeypatch):
    """The current stream's handle through torch's public interface."""
    asked = []

    def current_stream(device):
        asked.append(device)
        return SimpleNamespace(cuda_stream=1234)

    monkeypatch.setattr(torch.cuda, "current_stream", current_stream)
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    t = SimpleNamespace(is_cuda=True, device="cuda:3", get_device=lambda: 3)
    assert _lib.stream_of(t) == 1234 and asked == ["cuda:3"]
