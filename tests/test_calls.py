"""Prepared calls (instantmimic_b200/calls.py): reused for the same buffers, rebuilt when a
buffer is rebound, replaced in place or gone, and no buffer is kept alive."""

import copy
import gc
import weakref
from types import SimpleNamespace

import torch

from instantmimic_b200 import _lib, calls


def _run(monkeypatch, owner, objs, extra=(), seen=None):
    monkeypatch.setattr(_lib, "lib", lambda: SimpleNamespace(stage=lambda *a: seen.append(a) or 0))
    monkeypatch.setattr(_lib, "current_stream_handle", lambda stream=None: 7)
    calls.call(owner, "stage", objs, extra, lambda: (tuple(o.data_ptr() for o in objs), None))


def test_a_call_is_prepared_once_per_set_of_buffers(monkeypatch):
    owner, seen = SimpleNamespace(), []
    a, b = torch.zeros(4), torch.ones(4)
    for _ in range(3):
        _run(monkeypatch, owner, (a, b), (1,), seen)
    assert seen == [(a.data_ptr(), b.data_ptr(), 7)] * 3
    first = owner._imn_calls["stage"]
    _run(monkeypatch, owner, (a, b), (1,), seen)
    assert owner._imn_calls["stage"] is first
    _run(monkeypatch, owner, (a, b), (2,), seen)  # another plain value
    assert owner._imn_calls["stage"] is not first
    c = torch.zeros(4)
    _run(monkeypatch, owner, (a, c), (2,), seen)  # rebound
    assert seen[-1] == (a.data_ptr(), c.data_ptr(), 7)
    c.data = torch.zeros(8)  # the same object names other memory now
    _run(monkeypatch, owner, (a, c), (2,), seen)
    assert seen[-1] == (a.data_ptr(), c.data_ptr(), 7)
    assert len(copy.deepcopy(owner)._imn_calls) == 0


def test_a_prepared_call_keeps_no_buffer(monkeypatch):
    owner, seen = SimpleNamespace(), []
    a, b = torch.zeros(4), torch.ones(4)
    _run(monkeypatch, owner, (a, b), (), seen)
    gone = weakref.ref(b)
    del b
    gc.collect()
    assert gone() is None and not owner._imn_calls["stage"].alive
