"""The ring of pinned staging buffers (CPU, with stand-ins for pinned memory and events)."""
import threading

import pytest
import torch

from xinfer_b200.parts.attention_backend import PinnedRing


class _Event:
    made = []

    def __init__(self):
        self.recorded = self.waited = 0
        _Event.made.append(self)

    def record(self):
        self.recorded += 1

    def synchronize(self):
        self.waited += 1


@pytest.fixture(autouse=True)
def _stand_ins(monkeypatch):
    _Event.made = []
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda t: t)
    monkeypatch.setattr(torch.cuda, "Event", _Event)


def test_a_buffer_is_taken_again_only_after_its_event():
    ring = PinnedRing()
    seen = []
    for n in (10, 10, 10, 10, 10):
        seen.append(ring.take(n).data_ptr())
        ring.sent()
    assert len(set(seen[:4])) == 4 and seen[4] == seen[0]
    assert [e.waited for e in _Event.made] == [1, 0, 0, 0, 0]
    assert ring.take(100_000).numel() >= 100_000


def test_threads_do_not_take_each_others_buffers():
    ring = PinnedRing()
    mine = ring.take(10)
    others = []

    def other():
        for _ in range(9):
            others.append(ring.take(10))
            ring.sent()
    t = threading.Thread(target=other)
    t.start()
    t.join()
    assert mine.data_ptr() not in {b.data_ptr() for b in others}
    ring.sent()
    for _ in range(3):
        assert ring.take(10).data_ptr() != mine.data_ptr()
        ring.sent()
    last = _Event.made[9]           # the event of the buffer taken first
    assert last.waited == 0 and ring.take(10).data_ptr() == mine.data_ptr() and last.waited == 1
