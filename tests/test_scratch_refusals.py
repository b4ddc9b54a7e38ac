"""Scratch of the two-launch linear on a device without room for it: one refusal, not one per call. On the CPU, with the
allocator and the count of free bytes replaced."""
import pytest
import torch

from mflux_b200 import ops


class _Device:
    """`free` bytes left; requests are counted, those of more than is free are refused."""

    index = 0

    def __init__(self, monkeypatch, free):
        self.free, self.asked, self.capturing = free, [], False
        monkeypatch.setattr(ops, "_REFUSED", {})
        monkeypatch.setattr(ops, "_free_bytes", lambda device: self.free)
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: self.capturing)
        monkeypatch.setattr(torch, "empty", self._empty)

    def _empty(self, size, **kw):
        self.asked.append(size)
        if size > self.free:
            raise torch.OutOfMemoryError("no room")
        return size


def test_a_refused_size_is_not_asked_for_on_every_call(monkeypatch):
    d = _Device(monkeypatch, 100)
    assert [ops._scratch(size, d) for size in (300, 300, 400, 300)] == [None] * 4
    assert d.asked == [300]
    assert ops._scratch(80, d) == 80 and d.asked == [300, 80]       # smaller ones still are


def test_it_is_asked_for_again_once_more_is_free(monkeypatch):
    d = _Device(monkeypatch, 100)
    ops._scratch(300, d)
    d.free = 250                                   # more than then, but still no room: refused once more
    ops._scratch(300, d)
    for d.free in (200, 250):                      # what temporaries of a step come and go with
        assert ops._scratch(300, d) is None
    assert d.asked == [300, 300]
    d.free = 1000
    assert ops._scratch(300, d) == 300 and ops._REFUSED == {0: {}}
    assert ops._scratch(300, d) == 300


def test_no_question_to_the_driver_while_a_graph_is_captured(monkeypatch):
    d = _Device(monkeypatch, 100)
    ops._scratch(300, d)
    d.capturing, d.free = True, 1000
    monkeypatch.setattr(ops, "_free_bytes", lambda device: pytest.fail("asked during a capture"))
    assert ops._scratch(300, d) is None and ops._scratch(50, d) == 50


def test_the_record_is_bounded(monkeypatch):
    d = _Device(monkeypatch, 10)
    for size in range(1000, 1, -1):
        ops._scratch(size, d)
    assert len(ops._REFUSED[0]) <= 64
