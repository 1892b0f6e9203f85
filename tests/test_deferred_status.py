"""Deferred status words: waiting for a call waits for that call alone, and captured calls take no slot."""
import ctypes
import threading
import time

import pytest
import torch

import flashlib_b200 as fl
from flashlib_b200 import _lib
from flashlib_b200 import knn as knn_mod


def _slot(words):
    slot = object.__new__(knn_mod._StatusSlot)
    slot.buf, slot.ptr, slot.device = None, 0, torch.device("cuda", 0)
    slot.words = (ctypes.c_int32 * (_lib.FL_STATUS_WORDS + 1))(*words)
    return slot


@pytest.fixture
def queues(monkeypatch):
    from collections import deque
    monkeypatch.setattr(knn_mod, "_PENDING_STATUS", deque())
    monkeypatch.setattr(knn_mod, "_FREE_SLOTS", deque())

    def no_wait(*a, **k):
        raise AssertionError("a wait for the whole device")

    monkeypatch.setattr(torch.cuda, "synchronize", no_wait)


def test_waits_for_the_mark_of_the_call(queues):
    slot = _slot([0] * (_lib.FL_STATUS_WORDS + 1))
    knn_mod._PENDING_STATUS.append(slot)
    knn_mod.check_pending(block=False)
    assert len(knn_mod._PENDING_STATUS) == 1

    def finish():
        time.sleep(0.05)
        slot.words[_lib.FL_STATUS_ERROR] = _lib.FL_ETIMEOUT
        slot.words[_lib.FL_STATUS_WORDS] = 1

    t = threading.Thread(target=finish)
    t.start()
    with pytest.raises(_lib.FlashlibError):
        knn_mod.check_pending()
    t.join()
    assert not knn_mod._PENDING_STATUS and len(knn_mod._FREE_SLOTS) == 1


def test_a_failed_device_ends_the_wait(queues, monkeypatch):
    class Stream:
        def query(self):
            raise RuntimeError("CUDA error")

    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: Stream())
    knn_mod._PENDING_STATUS.append(_slot([0] * (_lib.FL_STATUS_WORDS + 1)))
    with pytest.raises(RuntimeError):
        knn_mod.check_pending()


@pytest.mark.gpu
def test_other_streams_are_not_waited_for():
    g = torch.Generator().manual_seed(1)
    db, q = torch.randn(30_000, 32, generator=g).cuda(), torch.randn(600, 32, generator=g).cuda()
    fl.flash_knn(q, db, 5)
    fl.check_pending()
    torch.cuda.synchronize()
    other = torch.cuda.Stream()
    with torch.cuda.stream(other):
        torch.cuda._sleep(1_000_000_000)            # half a second of one thread's time
    for _ in range(100):
        fl.flash_knn(q, db, 5)
    fl.check_pending()
    assert not other.query()
    torch.cuda.synchronize()


@pytest.mark.gpu
def test_captured_calls_take_no_slot():
    g = torch.Generator().manual_seed(2)
    db, q = torch.randn(30_000, 32, generator=g).cuda(), torch.randn(600, 32, generator=g).cuda()
    warm = torch.cuda.Stream()
    with torch.cuda.stream(warm):
        for _ in range(3):
            fl.flash_knn(q, db, 5)
    fl.check_pending()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        vals, idxs = fl.flash_knn(q, db, 5)
    assert not knn_mod._PENDING_STATUS
    q.copy_(torch.randn(600, 32, generator=g))
    graph.replay()
    want_v, want_i = fl.flash_knn(q, db, 5)
    graph.replay()
    fl.check_pending()
    assert torch.equal(vals, want_v) and torch.equal(idxs, want_i)
