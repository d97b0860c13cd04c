"""What the autotuner may choose: knobs of the tile kernels, and nothing where
the block kernels run, which take none (no GPU: times and launches are stood
in for)."""
import pytest
import torch

from gstex_cuda_gb300 import batch as B


@pytest.fixture(autouse=True)
def _stand_in(monkeypatch):
    class Event:
        def __init__(self, enable_timing=False):
            pass

        def record(self, stream):
            pass

        def elapsed_time(self, other):
            Event.ms += 1.0  # later candidates look slower ...
            return 1000.0 - Event.ms if Event.falling else Event.ms  # ... or faster

    Event.ms, Event.falling = 0.0, True
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: None)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda dev=None: None)
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda dev=None: "GB300")
    monkeypatch.delenv("GSTEX_AUTOTUNE_CACHE", raising=False)
    monkeypatch.setattr(B, "_tune_cache", {})


def _renderer(records=True, bw=8, channels=3, settings=1 << 8, **knobs):
    """The parts of a BatchRenderer that the autotuner reads; launches are counted."""
    r = object.__new__(B.BatchRenderer)
    r.sizes, r.N, r.C, r.texmode, r.settings, r.bw, r.dev = [(64, 64)], 100, channels, 1, settings, bw, "cuda:0"
    r.records = object() if records else None
    r.fwd_ppt, r.fwd_batch, r.bwd_ppt, r.bwd_group, r.bwd_ctas, r.bwd_batch = 1, 0, 1, 8, 0, 0
    for k, v in knobs.items():
        setattr(r, k, v)
    r.graph, r.calls = None, []
    r.bin = lambda s: None
    r.forward = lambda s: r.calls.append("forward")
    r.backward = lambda s: r.calls.append("backward")
    r.image_loss = lambda *t: None
    return r


def _knobs(r):
    return {k: getattr(r, k) for k in B.TUNED_KNOBS}


def test_block_kernels_are_timed_once_and_keep_the_knobs():
    r = _renderer(bwd_group=32, bwd_batch=48)
    before = _knobs(r)
    assert not r.takes_knobs()
    res = r.autotune(None, None, None, reps=1)
    assert _knobs(r) == before and res["bwd_group"] == 32
    # (one warm-up and one timed launch each, and the forward whose loss the backward takes)
    assert r.calls.count("forward") == 3 and r.calls.count("backward") == 2
    assert len({v for k, v in res.items() if k.startswith("backward") and k.endswith("_ms")}) == 1
    assert {"forward_ppt1_ms", "forward_ppt2_ms", "backward_ppt1_g8_ms", "backward_ppt1_g8_ctas10_ms"} <= set(res)
    again = _renderer(bwd_group=16)
    assert again.autotune(None, None, None)["cached"] and not again.calls and again.bwd_group == 16


@pytest.mark.parametrize("kw", [dict(records=False), dict(channels=4), dict(bw=12), dict(settings=(1 << 8) | (1 << 16))])
def test_tile_kernels_are_tuned_as_before(kw):
    r = _renderer(**kw)
    assert r.takes_knobs()
    res = r.autotune(None, None, None, reps=1)
    assert len({v for k, v in res.items() if k.endswith("_ms")}) == len([k for k in res if k.endswith("_ms")])
    assert _knobs(r)["fwd_ppt"] == (2 if r.bw * r.bw <= 64 else 1)  # (the last candidate looked fastest)
    again = _renderer(**kw)
    assert again.autotune(None, None, None)["cached"] and _knobs(again) == _knobs(r)


def test_kernels_do_not_take_each_others_tunings():
    """Block and tile kernels of one configuration have keys of their own, and
    neither takes an entry without one; configurations that only the tile
    kernels serve keep the plain key, with or without records."""
    for bw, C, s, own in ((8, 3, 256, True), (16, 0, 0, True), (8, 4, 256, False), (12, 3, 256, False),
                          (16, 3, 1 << 16, False)):
        a, b = (_renderer(rec, bw, C, s).tune_key() for rec in (True, False))
        plain = B.autotune_key([(64, 64)], 100, C, 1, s, bw, "GB300")
        assert (a != b) is own and (plain in (a, b)) is not own
