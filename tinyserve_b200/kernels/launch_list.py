"""The launches of layers that differ in nothing but their tensors, run from the library (``csrc/launch_list.cu``).

A step that is not replayed from a recording is launched kernel by kernel, 14 to 17 us of the host's time each, most of it
spent in the interpreter on checks and choices that come out the same for every layer. So the model runs the first layers
of such a row as always, writes down what two neighbouring ones launched, and hands that over for all further ones: the
library makes the same calls with each pointer into one of the layer's own tensors moved to the next layer's. No list is
kept from one step for the next; where the layers' tensors lie is known from when they were bound, and looked at again for
every list.
"""

from __future__ import annotations

import ctypes
import functools
import struct
from array import array
from typing import Any, Sequence

from . import build, ops

_FORMATS = {ctypes.c_void_p: "Q", ctypes.c_int: "q", ctypes.c_longlong: "q", ctypes.c_ulonglong: "Q", ctypes.c_size_t: "Q",
            ctypes.c_float: "f4x", ctypes.c_double: "d"}


_KINDS = {ctypes.c_void_p: "p", ctypes.c_int: "i", ctypes.c_longlong: "l", ctypes.c_ulonglong: "l", ctypes.c_size_t: "l",
          ctypes.c_float: "f", ctypes.c_double: "d"}


@functools.lru_cache(maxsize=None)
def _entry(name: str) -> "tuple[int, struct.Struct] | None":
    """The entry point's number in the library's table and the layout of its arguments; ``None``: no list may name it."""
    lib = build.library()
    lib.ts_list_entry.argtypes, lib.ts_list_entry.restype = [ctypes.c_char_p, ctypes.c_void_p, ctypes.c_void_p], ctypes.c_int
    count, kinds = ctypes.c_int(0), ctypes.create_string_buffer(65)
    number = lib.ts_list_entry(name.encode(), ctypes.addressof(count), ctypes.addressof(kinds))
    if number < 0:
        return None
    types = ops._SIGNATURES[name]
    if kinds.value.decode() != "".join(_KINDS[t] for t in types):
        raise ops.KernelError(f"{name}: the library's arguments are {kinds.value.decode()}")
    return number, struct.Struct("<" + "".join(_FORMATS[t] for t in types))


@functools.lru_cache(maxsize=None)
def _run() -> Any:
    f = build.library().ts_list_run
    f.argtypes, f.restype = [ctypes.c_void_p] * 5 + [ctypes.c_int, ctypes.c_int, ctypes.c_void_p], ctypes.c_int
    return f


class Noting:
    """While it is open, this thread's calls of the library are kept in ``calls``, and ``kernels`` counts the launches."""

    def __enter__(self) -> "Noting":
        self.calls: list[tuple[str, tuple[Any, ...]]] = []
        self.kernels = -ops.launch_count
        self._outer, ops.notes.calls = ops.notes.calls, self.calls
        return self

    def __exit__(self, *exc: Any) -> None:
        ops.notes.calls = self._outer
        self.kernels += ops.launch_count


_UNLIKE = -4


def run(noted: "Sequence[Noting]", places: "array[int]", sizes: "list[int]") -> bool:
    """The launches of further layers. ``noted``: those of two neighbouring layers; ``places``: where the tensors of each
    layer lie, of the two first and then of the layers to run, which take turns at the two; ``sizes``: the bytes of a
    layer's tensors. False (and nothing is launched) if a call is none that a list may hold, or if a layer's
    tensors lie differently to the 16-byte grid that the kernels choose their accesses by."""
    entries, words, first = [], [], [0]
    for n in noted:
        for name, args in n.calls:
            e = _entry(name)
            if e is None:
                return False
            entries.append(e[0])
            try:
                words.append(e[1].pack(*[a or 0 for a in args]))
            except struct.error:          # an argument that is no plain number
                return False
        first.append(len(entries))
    layers = len(places) // len(sizes) - 2
    numbers, firsts, nbytes, failed = array("i", entries), array("i", first), array("Q", sizes), array("i", [0, 0])
    status = _run()(numbers.buffer_info()[0], firsts.buffer_info()[0], b"".join(words), places.buffer_info()[0],
                    nbytes.buffer_info()[0], len(sizes), layers, failed.buffer_info()[0])
    if status == _UNLIKE:
        return False
    if status != 0:
        calls = noted[0].calls + noted[1].calls
        ops._check(status, f"layer {failed[0]} of a list of launches, {calls[failed[1]][0]}")
    ops.launch_count += (layers + 1) // 2 * noted[0].kernels + layers // 2 * noted[1].kernels
    return True
