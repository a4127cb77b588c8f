"""Prepared C-ABI calls.

A step pipeline calls the same stages with the same buffers every substep, and building a
call's structs (attribute walks, stride and shape checks) takes longer than the GPU needs for
a small batch.  The structs are therefore built once per set of buffers and kept on the object
that owns the buffers (a ``Data`` or a scratch).  Every later call compares the buffers with
the ones the structs were built from -- the very objects, and the address each of them names
now -- and builds anew when one differs.  A prepared call keeps no buffer alive.
"""

from __future__ import annotations

from operator import attrgetter
from typing import Any, Callable
from weakref import ref

from . import _lib
from .arrays import addr

_data_ptr = None


def pointers(objs: tuple) -> tuple:
    """The addresses of a tuple of arrays (torch tensors in one pass, others one by one)."""
    global _data_ptr
    if _data_ptr is None:
        import torch

        _data_ptr = torch.Tensor.data_ptr
    try:
        return tuple(map(_data_ptr, objs))
    except TypeError:
        return tuple(map(addr, objs))


def optional_pointers(objs: tuple) -> tuple:
    """The same where arrays may be missing (None)."""
    try:
        return tuple([None if o is None else o.data_ptr() for o in objs])
    except AttributeError:
        return tuple(map(addr, objs))


class CallCache(dict):
    """The prepared calls of one owner, by stage; a copy of the owner starts without any."""

    def __deepcopy__(self, memo):
        return CallCache()

    def __reduce__(self):
        return (CallCache, ())


class Prepared:
    __slots__ = ("alive", "refs", "ids", "ptrs", "extra", "fn", "args", "what", "keep")

    def __init__(self, what: str, objs: tuple, extra: tuple, fn: Callable, args: tuple, keep: Any):
        self.what, self.extra, self.fn, self.args, self.keep = what, extra, fn, args, keep
        self.ids, self.ptrs = tuple(map(id, objs)), pointers(objs)
        # empty once one of the objects is gone: its id may then name another one
        self.alive = alive = [True]
        try:
            self.refs = [ref(o, lambda _, alive=alive: alive.clear()) for o in objs if o is not None]
        except TypeError:  # an array type that cannot be watched: built anew every time
            alive.clear()

    def __call__(self, stream=None) -> None:
        if _lib.nvtx_enabled():
            with _lib.nvtx(self.what):
                rc = self.fn(*self.args, _lib.current_stream_handle(stream))
        else:
            rc = self.fn(*self.args, _lib.current_stream_handle(stream))
        if rc:
            _lib.check(rc, self.what)


def call(owner: Any, what: str, objs: tuple, extra: tuple, build: Callable[[], tuple], stream=None,
         slot: Any = None) -> None:
    """Run stage ``what`` on the buffers ``objs`` with the plain values ``extra``.  ``build``
    returns (arguments before the stream, what must stay alive with them).  ``slot`` tells calls of
    one stage apart that an owner makes in turn."""
    try:
        cache = owner.__dict__["_imn_calls"]
    except (AttributeError, KeyError):
        cache = CallCache()
        try:
            owner._imn_calls = cache
        except AttributeError:
            pass
    key = what if slot is None else (what, slot)
    p = cache.get(key)
    if p is None or not p.alive or p.ids != tuple(map(id, objs)) or p.extra != extra or p.ptrs != pointers(objs):
        args, keep = build()
        p = cache[key] = Prepared(what, objs, extra, getattr(_lib.lib(), what), args, keep)
    p(stream)


def getter(*names: str) -> Callable[[Any], tuple]:
    """Reads several (dotted) attributes at once; always a tuple."""
    if len(names) > 1:
        return attrgetter(*names)
    one = attrgetter(names[0])
    return lambda obj: (one(obj),)
