"""Scratch memory of a step: a bump allocator over buffers that are reused every step.

Three regions: ``step`` holds what lives for the whole step (the residual stream, position
tables, logits); two ``frames`` alternate from layer to layer, so that the output a layer
leaves pending on the residual stream is still intact while the next layer, working in the
other frame, reads it. Nothing is allocated from the device allocator in steady state; a
region grows (once, outside any graph capture) when a step needs more than it has.

The layers of a step ask for the same shapes at the same offsets, so a region keeps the views it
has made of its buffer (slicing and viewing took a quarter of the host's time for a step that is
launched kernel by kernel: 1.2 of 4.4 ms for 28 dense layers).
"""

from __future__ import annotations

import torch

_ALIGN = 256
_MOST_VIEWS = 1024      # kept per region; prompts of ever new lengths ask for ever new shapes
_ELEMENT_SIZE: dict[torch.dtype, int] = {}


def _element_size(dtype: torch.dtype) -> int:
    n = _ELEMENT_SIZE.get(dtype)
    if n is None:
        n = _ELEMENT_SIZE[dtype] = torch.empty(0, dtype=dtype).element_size()
    return n


class _Region:
    def __init__(self, device: torch.device) -> None:
        self.device = device
        self.buf = torch.empty(0, dtype=torch.uint8, device=device)
        self._typed: dict[torch.dtype, torch.Tensor] = {}     # ``buf`` seen as each dtype asked for so far
        # (offset, shape, dtype) -> (the view of ``buf`` handed out for it, its bytes)
        self._views: dict[tuple[int, tuple[int, ...], torch.dtype], tuple[torch.Tensor, int]] = {}
        self.used = 0          # offset in ``buf`` of the next take
        self.demand = 0        # bytes taken since the last reset, wherever they came from
        self.high_water = 0    # the largest demand of any step so far
        self.moves = 0         # how often ``buf`` has been made anew

    def reset(self) -> None:
        if self.high_water > self.buf.numel():
            # The last step outgrew the buffer and was served piecemeal; make one buffer that
            # holds a whole step, so that from now on nothing moves.
            self.buf = torch.empty(self.high_water // _ALIGN * _ALIGN + _ALIGN, dtype=torch.uint8, device=self.device)
            self.moves += 1
            self._typed = {}
            self._views = {}
        elif len(self._views) > _MOST_VIEWS:
            self._views = {}
        self.used = 0
        self.demand = 0

    def take(self, shape: tuple[int, ...], dtype: torch.dtype) -> torch.Tensor:
        start = (self.used + _ALIGN - 1) // _ALIGN * _ALIGN
        made = self._views.get((start, shape, dtype))
        if made is not None:
            self.demand = (self.demand + _ALIGN - 1) // _ALIGN * _ALIGN + made[1]
            if self.demand > self.high_water:
                self.high_water = self.demand
            self.used = start + made[1]
            return made[0]
        numel = 1
        for s in shape:
            numel *= int(s)
        size = _element_size(dtype)
        nbytes = numel * size
        before = self.demand, self.high_water
        self.demand = (self.demand + _ALIGN - 1) // _ALIGN * _ALIGN + nbytes
        self.high_water = max(self.high_water, self.demand)
        end = start + nbytes
        if end > self.buf.numel():
            # Grow: views handed out earlier keep the old buffer alive until they die.
            grow = max(nbytes, 2 * self.buf.numel(), 1 << 16)
            try:
                self.buf = torch.empty((grow + _ALIGN - 1) // _ALIGN * _ALIGN, dtype=torch.uint8, device=self.device)
            except torch.cuda.OutOfMemoryError:
                self.demand, self.high_water = before        # who can do without it goes on; no later step is to hold it
                raise
            self.moves += 1
            self._typed = {}
            self._views = {}
            start, end = 0, nbytes
        self.used = end
        if numel == 0:
            return torch.empty(shape, dtype=dtype, device=self.device)
        typed = self._typed.get(dtype)
        if typed is None:
            typed = self._typed[dtype] = self.buf.view(dtype)     # buffer sizes are multiples of 256 bytes
        view = typed[start // size: end // size].view(shape)
        self._views[(start, shape, dtype)] = (view, nbytes)
        return view


class Arena:
    def __init__(self, device: torch.device | str) -> None:
        self.device = torch.device(device)
        self._step = _Region(self.device)
        self._frames = (_Region(self.device), _Region(self.device))
        self._current = self._step
        self._frame_index = 0

    def begin_step(self) -> None:
        self._step.reset()
        for f in self._frames:
            f.reset()
        self._current = self._step
        self._frame_index = 0

    def next_frame(self) -> None:
        self._frame_index ^= 1
        self._current = self._frames[self._frame_index]
        self._current.reset()

    def frame_state(self) -> tuple[int, int, int]:
        """The current frame and how far it is used, for ``resume_frame``."""
        return self._frame_index, self._current.used, self._current.demand

    def resume_frame(self, state: tuple[int, int, int]) -> None:
        """The frame of ``state`` again, used as far as it was then: what was taken from it stays whole. (``next_frame`` hands
        a frame over empty.)"""
        self._frame_index, used, demand = state
        self._current = self._frames[self._frame_index]
        self._current.used, self._current.demand = used, demand

    def step_region(self) -> None:
        """Later takes live until the end of the step (used after the last layer)."""
        self._current = self._step

    def take(self, shape: tuple[int, ...], dtype: torch.dtype) -> torch.Tensor:
        return self._current.take(tuple(shape), dtype)

    def take_step(self, shape: tuple[int, ...], dtype: torch.dtype) -> torch.Tensor:
        return self._step.take(tuple(shape), dtype)

    @property
    def moves(self) -> int:
        """Grows whenever a region's buffer is made anew (what was handed out before then lies elsewhere)."""
        return self._step.moves + sum(f.moves for f in self._frames)

    @property
    def reserved_bytes(self) -> int:
        return self._step.buf.numel() + sum(f.buf.numel() for f in self._frames)
