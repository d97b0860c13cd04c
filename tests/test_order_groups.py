"""Host side of the forward's queue order (no GPU: nothing is launched)."""
import ctypes

import pytest
import torch

from gstex_cuda_gb300 import batch as B


def _renderer(width, height, group):
    """The parts of a BatchRenderer that its tile groups are made of, on the CPU."""
    r = object.__new__(B.BatchRenderer)
    r.descs = (B.ViewDesc * 1)()
    r.descs[0].fx = r.descs[0].fy = 1.0
    r.descs[0].width, r.descs[0].height = width, height
    r.V, r.bw, r.order_group, r.dev = 1, 8, group, torch.device("cpu")
    r._order_groups = {}
    return r


def test_groups_of_an_earlier_order_group_stay(monkeypatch):
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    r = _renderer(40, 24, 4)
    first = r._tile_groups()
    assert first.tolist() == [[0, 5, 4, 3], [4, 5, 1, 3]]
    r.order_group = 2
    assert r._tile_groups().shape[0] == 6
    r.order_group = 4
    assert r._tile_groups() is first
    r.order_group = 3
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert r._tile_groups() is None


@pytest.mark.parametrize("group,ok", [(-1, False), (0, False), (1, True), (64, True), (65, False), (1000, False)])
def test_order_groups_that_are_refused(group, ok, monkeypatch):
    """1 to 64 tiles a side, as gstex_batch_tile_order takes them; others have
    no groups, and the renderer's step goes on to the refusal there."""
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    r = _renderer(40, 24, group)
    rows, n = torch.empty((64, 4), dtype=torch.int32), ctypes.c_int(0)
    rc = B._L().gstex_batch_tile_groups(1, r.descs, 8, group, 64, rows.data_ptr(), ctypes.byref(n))
    assert rc == (0 if ok else 1) and (r._tile_groups() is not None) is ok
