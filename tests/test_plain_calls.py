"""Which calls a kernel launch may stand for (no GPU: tensors and torch's answers
are stood in for)."""
from types import SimpleNamespace

import pytest
import torch

from gstex_cuda_gb300 import _lib


class Plain:
    """The parts of a tensor that plain_cuda_f32 reads."""
    is_cuda, dtype, requires_grad, layout = True, torch.float32, False, torch.strided

    def __init__(self, device=0, negated=False, **parts):
        self.device, self.negated = device, negated
        self.__dict__.update(parts)

    def is_neg(self):
        return self.negated

    def get_device(self):
        return self.device


@pytest.fixture
def plain(monkeypatch):
    """plain_cuda_f32 for stand-in tensors on a machine whose current device is 0."""
    monkeypatch.setattr(torch, "Tensor", Plain)
    monkeypatch.setattr(_lib, "_current_device", lambda: 0)
    return _lib.plain_cuda_f32


def test_plain_tensors(plain):
    assert plain(Plain(), Plain())


@pytest.mark.parametrize("places,current,want", [((0,), 0, True), ((1,), 0, False), ((1, 1), 1, True),
                                                 ((0, 1), 0, False), ((0, 1), 1, False)])
def test_launches_go_to_the_current_device(places, current, want, plain, monkeypatch):
    """A launch goes to the current device, so tensors of another one keep the
    torch operations, which go to theirs."""
    monkeypatch.setattr(_lib, "_current_device", lambda: current)
    assert plain(*(Plain(p) for p in places)) is want


@pytest.mark.parametrize("parts", [dict(is_cuda=False), dict(dtype=torch.float16), dict(requires_grad=True),
                                   dict(layout=torch.sparse_coo), dict(negated=True)])
def test_other_tensors(parts, plain):
    assert not plain(Plain(), Plain(**parts)) and not plain(Plain(**parts), Plain())
    with torch.no_grad():
        assert plain(Plain(), Plain(**parts)) is ("requires_grad" in parts)


def test_projection_asks(monkeypatch):
    """project_points asks before it launches."""
    from gstex_cuda_gb300 import get_aabb_2d as A
    seen = []
    monkeypatch.setattr(_lib, "plain_cuda_f32", lambda *t: seen.append(len(t)))
    pix, depth = A.project_points(torch.ones(3, 3), torch.eye(4), (1.0, 1.0, 0.0, 0.0))
    assert seen == [2] and depth.tolist() == [1.0, 1.0, 1.0]


def test_products_in_another_type(plain, monkeypatch):
    """Autocast and torch's reduced-precision products change the torch
    operations' results; a launch, which computes in float32, does not stand
    for them then."""
    with monkeypatch.context() as m:
        m.setattr(_lib, "_autocast", lambda device: device == "cuda")
        assert not plain(Plain())
    for precision in ("high", "medium"):
        monkeypatch.setattr(_lib, "_precision", lambda: precision)
        assert not plain(Plain())

    def mixed():
        raise RuntimeError("set through both interfaces")

    monkeypatch.setattr(_lib, "_precision", mixed)
    assert not plain(Plain())


def test_observers(plain, monkeypatch):
    """Anything that looks at torch operations: a compiler, a forward-mode
    level, a functional transform, a tracer, a dispatch or function mode."""
    with monkeypatch.context() as m:
        m.setattr(_lib, "_is_compiling", lambda: True)
        assert not plain(Plain())
    with torch.autograd.forward_ad.dual_level():
        assert not plain(Plain())
    quiet = (lambda: None, lambda: None, lambda: 0, lambda: 0)
    for k in range(4):
        ask = list(quiet)
        ask[k] = lambda: 1
        monkeypatch.setattr(_lib, "_questions", tuple(ask))
        assert not plain(Plain())
    monkeypatch.setattr(_lib, "_questions", quiet)
    assert plain(Plain())


@pytest.mark.parametrize("name", ["_functorch", "_get_tracing_state", "_len_torch_dispatch_stack",
                                  "_len_torch_function_stack"])
def test_a_torch_without_one_of_its_private_names(name, plain, monkeypatch):
    """Names that torch does not promise: without one the torch operations are
    kept."""
    names = ("_functorch", "_get_tracing_state", "_len_torch_dispatch_stack", "_len_torch_function_stack")
    assert _lib.private_questions() is not None
    without = SimpleNamespace(**{n: getattr(torch._C, n) for n in names if n != name})
    assert _lib.private_questions(without) is None
    monkeypatch.delattr(torch.autograd.forward_ad, "_current_level")
    assert _lib.private_questions() is None
    monkeypatch.undo()
    monkeypatch.setattr(torch, "Tensor", Plain)
    monkeypatch.setattr(_lib, "_current_device", lambda: 0)
    monkeypatch.setattr(_lib, "_questions", None)
    assert not _lib.plain_cuda_f32(Plain())


def test_streams_without_the_raw_lookup(monkeypatch):
    """The current stream's handle through torch's public interface."""
    asked = []

    def current_stream(device):
        asked.append(device)
        return SimpleNamespace(cuda_stream=1234)

    monkeypatch.setattr(torch.cuda, "current_stream", current_stream)
    monkeypatch.setattr(_lib, "_raw_stream", None)
    t = SimpleNamespace(is_cuda=True, device="cuda:3", get_device=lambda: 3)
    assert _lib.stream_of(t) == 1234 and asked == ["cuda:3"]
