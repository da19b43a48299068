"""Pinned staging buffers outlive the copies that read them, and a group drops only its own launch plans."""
import gc

import pytest
import torch

from adafactor8bit import _engine as E


class FakeEvent:
    """An event that has passed when `done` is set; `on_query` runs at the next query."""

    def __init__(self):
        self.done, self.on_query = False, None

    def record(self, stream):
        self.done = False

    def query(self):
        hook, self.on_query = self.on_query, None
        if hook:
            hook()
        return self.done

    def synchronize(self):
        self.done = True


@pytest.fixture
def ring(monkeypatch):
    """A function that makes rings of pageable memory with fake events."""
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, pin_memory=False, **kw: empty(*a, **kw))
    monkeypatch.setattr(torch.cuda, "Event", FakeEvent)
    E._RETIRED.clear()
    yield lambda: E._PinnedRing(64)
    E._RETIRED.clear()


def used(ring):
    """-> (buffer address, event) of the ring's next buffer, with a copy queued."""
    ring.next()
    ring.mark(None)
    return ring.bufs[ring.i].data_ptr(), ring.events[ring.i]


def test_a_dropped_ring_keeps_the_buffers_of_queued_copies(ring):
    r = ring()
    first, second = used(r), used(r)
    first[1].done = True
    del r
    gc.collect()
    assert [b.data_ptr() for b, _ in E._RETIRED] == [second[0]]       # (the other copies are done, or there were none)
    keep = ring()
    assert len(E._RETIRED) == 1                                       # still queued
    second[1].done = True
    more = ring()
    assert len(E._RETIRED) == 0
    del keep, more


def test_a_ring_dropped_while_others_are_released_is_kept(ring):
    """By another thread, or by a collection that the release itself sets off."""
    r, late = ring(), [ring()]
    a, b = used(r), used(late[0])
    del r
    gc.collect()
    a[1].on_query = late.clear
    keep = ring()
    assert sorted(x.data_ptr() for x, _ in E._RETIRED) == sorted((a[0], b[0]))
    del keep


def test_an_event_that_cannot_be_asked_counts_as_pending(ring):
    r = ring()
    _, event = used(r)

    def fail():
        raise RuntimeError("not now")

    event.on_query = fail
    del r
    gc.collect()
    assert len(E._RETIRED) == 1


@pytest.mark.gpu
def test_a_group_drops_only_its_own_plans():
    from adafactor8bit import Adafactor8Bit
    params = [torch.nn.Parameter(torch.randn(4096, device="cuda")) for _ in range(2)]
    opt = Adafactor8Bit([dict(params=[params[0]]), dict(params=[params[1]])], beta1=0.9, beta2=0.999, factored=False)
    for p in params:
        p.grad = torch.randn_like(p)
    opt.step()
    before = dict(opt._plans)
    opt.param_groups[1]["m_quant_type"] = "uf4"
    opt.step()
    assert {k[0] for k in before} == {0, 1}
    assert all(opt._plans[k] is v for k, v in before.items() if k[0] == 0)
    assert all(opt._plans.get(k) is not v for k, v in before.items() if k[0] == 1)
    torch.cuda.synchronize()
