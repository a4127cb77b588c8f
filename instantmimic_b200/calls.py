"""C-ABI calls of the stage functions.

Every call reads the buffers it is given -- addresses, strides and what has to be checked -- and packs
its structs anew: nothing is kept from one call for the next, so a buffer that is rebound, reshaped in
place or gone is never met again, and threads share nothing.  Packing a struct's fields in one
pass takes less time than finding out whether they have changed (24 fields 0.24 us; the identities of
as many objects 0.8).
"""

from __future__ import annotations

from operator import attrgetter
from typing import Any, Callable

from . import _lib


def call(what: str, args: tuple, stream=None) -> None:
    """Run ``what`` with ``args`` (structs as packed bytes) on a stream."""
    if _lib.nvtx_enabled():
        with _lib.nvtx(what):
            rc = _lib.packed(what)(*args, _lib.current_stream_handle(stream))
    else:
        rc = _lib.packed(what)(*args, _lib.current_stream_handle(stream))
    if rc:
        _lib.check(rc, what)


def getter(*names: str) -> Callable[[Any], tuple]:
    """Reads several (dotted) attributes at once; always a tuple."""
    if len(names) > 1:
        return attrgetter(*names)
    one = attrgetter(names[0])
    return lambda obj: (one(obj),)
