"""The generic decoder: a model is the parts its ``ModelSpec`` names, run in the order the
spec lists. There is no per-architecture model class; an architecture is a typed
configuration that produces a spec (``tinyserve_b200.architectures``).

One forward pass (after upstream src/tinyserve/model.py:181-200): embed the step's tokens
into the 32-bit residual stream, run every call of the order through its block, select the
wanted rows, apply the final norm to those rows only and multiply by the output head into
32-bit logits.
"""

from __future__ import annotations

import weakref
from array import array
from dataclasses import dataclass
from itertools import chain
from operator import itemgetter
from pathlib import Path
from typing import Any, Mapping

import torch

from . import parts as _parts  # noqa: F401  (registers the built-in parts)
from .kernels import launch_list, ops
from .config.base import LayerSpec, ModelConfig, ModelSpec
from .parts.base import (
    BLOCKS, EMBEDDINGS, HEADS, NORMS, PART_FAMILIES, POSITION_ENCODINGS, STREAM_INPUTS,
    Block, CacheNeed, KVCacheEntry, PagedNeed, PositionEncoding, ResidualStream, StepContext, StreamInput, TensorSpec, Watched, launches_alike,
)
from .weights.loader import load_tensors, merge_specs
from .weights.random_init import random_bound_tensors

# Above this estimate of a layer's products (what the product of its tensors' bytes and the step's tokens comes to at the rates
# of many rows, in a microsecond) its launches are not made from a list.
LISTED_LAYER_US = 40.0
BYTE_TOKENS_PER_US = {torch.bfloat16: 1.4e9, torch.float32: 7.4e7}


@dataclass
class Layer(Watched):
    spec: LayerSpec
    block: Block
    position: PositionEncoding | None
    positions: dict[str, PositionEncoding]      # by mixer role, when the mixers have encodings of their own


_TENSORS = frozenset({torch.Tensor, torch.nn.Parameter})      # (other classes of tensors are in no list)
_PLAIN = frozenset({bool, int, float, str, type(None)})


class _RowPlaces:
    """Where the tensors of a row of layers lie, call by call, and the bytes of each of a call's; with it, all that this was
    read from, so that whatever has been replaced since (a tensor, its storage, an attribute, a part) shows."""

    def __init__(self, layers: "list[Layer]", watched: list[dict[str, Any]], places: list[int], sizes: list[int]) -> None:
        self.places, self.sizes = places, sizes
        self._watched, self._layers, self._gone, self._seen, self._layer_ids = watched, layers, [], -1, list(map(id, layers))
        if not places:          # (a copy)
            self._gone.append(None)
            return
        values = self._values()
        types = list(map(type, values))
        tensors = [i for i, t in enumerate(types) if t in _TENSORS]
        self._tensors, self._others = itemgetter(*tensors), itemgetter(*[i for i, t in enumerate(types) if t not in _TENSORS])
        # tensors by their identity, which something new may have once one has gone: that is noted, so none is kept alive here
        self._ids = list(map(id, self._tensors(values)))
        self._alive = [weakref.ref(v, self._gone.append) for v in self._tensors(values)]
        self._plain, self._count = self._others(values), len(values)

    def _values(self) -> list[Any]:
        return list(chain(self._layers, *map(dict.values, self._watched)))

    def __reduce__(self) -> Any:      # a copy of the layers has them elsewhere: nothing holds for it, and it looks anew
        return _RowPlaces, ([], [], [], self.sizes)

    def hold(self) -> bool:
        if self._gone:
            return False
        changes = Watched.changes()
        if self._seen != changes or list(map(id, self._layers)) != self._layer_ids:
            values = self._values()
            if len(values) != self._count:
                return False
            try:
                if list(map(id, self._tensors(values))) != self._ids or self._others(values) != self._plain:
                    return False
            except (RuntimeError, ValueError):          # a tensor or an array where none was does not compare
                return False
            self._seen = changes
        return list(map(torch.Tensor.data_ptr, [t() for t in self._alive])) == self.places


class ModelParts:
    """The parts of a model, built from a spec but not yet holding weights."""

    def __init__(self, spec: ModelSpec) -> None:
        self.spec = spec
        self.embedding = EMBEDDINGS.build(spec.embedding.kind, **spec.embedding.args)
        self.final_norm = NORMS.build(spec.final_norm.kind, **spec.final_norm.args)
        self.head = HEADS.build(spec.head.kind, **spec.head.args)
        self._positions: dict[Any, PositionEncoding] = {}
        self.layers: list[Layer] = []
        for n, ls in enumerate(spec.layers):
            block = self._build_block(n, ls)
            pos = None if ls.position is None else self._encoding(ls.position)
            unknown = set(ls.positions) - set(block.mixers())
            if unknown:
                raise ValueError(f"layer {n}: position encodings for {sorted(unknown)}, which are no mixers of its block")
            self.layers.append(Layer(ls, block, pos, {role: self._encoding(p) for role, p in ls.positions.items()}))
        self.stream_inputs: list[StreamInput | None] = [
            None if c.stream_input is None else STREAM_INPUTS.build(c.stream_input.kind, **c.stream_input.args) for c in spec.order]
        for n, (call, part) in enumerate(zip(spec.order, self.stream_inputs)):
            block = self.layers[call.layer].block
            first_norm = next((block.parts[r] for r, family in type(block).roles.items() if family == "norm" and r in block.parts), None)
            if part is not None and not part.replaces and not getattr(first_norm, "folds_stream_input", False):
                raise ValueError(f"order[{n}] has a stream input, but the first norm of its block does not add it")
        self.keeps_origin = any(s is not None and s.needs_origin for s in self.stream_inputs)
        # One cache user per (call of the order, mixer role of its block, need of that mixer), in that order: the
        # cache manager gets their needs as a flat list and hands back one entry for each.
        self.cache_users: list[tuple[int, str]] = []
        self._user_index: dict[tuple[int, str], "int | tuple[int, ...]"] = {}
        self._needs: list[CacheNeed | None] = []
        for n, call in enumerate(spec.order):
            for role, mixer in self.layers[call.layer].block.mixers().items():
                need = mixer.cache_need()
                several = need if isinstance(need, tuple) else (need,)
                first = len(self.cache_users)
                self.cache_users += [(n, role)] * len(several)
                self._user_index[(n, role)] = tuple(range(first, first + len(several))) if isinstance(need, tuple) else first
                self._needs += several if call.reads_cache_of is None else (None,) * len(several)
        self._check_order()
        self._rows_of_alike = self._find_alike()
        self._row_places: "dict[int, _RowPlaces | None]" = {}      # of a row, once its parts hold their tensors
        self._cache_indices = []      # of a call: the cache entries that its mixers keep
        for n, call in enumerate(spec.order):
            of = [self._user_index[(n, role)] for role in self.layers[call.layer].block.mixers()]
            self._cache_indices.append([i for index in of for i in (index if isinstance(index, tuple) else (index,))
                                        if self._needs[i] is not None])

    def _encoding(self, spec: Any) -> PositionEncoding:
        cand = POSITION_ENCODINGS.build(spec.kind, **spec.args)
        return self._positions.setdefault(cand.key(), cand)

    @staticmethod
    def _build_block(n: int, ls: LayerSpec) -> Block:
        """The block class names its roles; every role is built from the registry of its family."""
        block_cls = BLOCKS.get(ls.block)
        roles = getattr(block_cls, "roles", None)
        if not roles:
            raise TypeError(f"block {ls.block!r} names no roles (a Block subclass with a ``roles`` mapping is needed)")
        optional = getattr(block_cls, "optional_roles", frozenset())
        unknown = set(ls.parts) - set(roles)
        missing = set(roles) - set(ls.parts) - set(optional)
        if unknown or missing:
            raise ValueError(f"layer {n} ({ls.block!r}): parts for unknown roles {sorted(unknown)}, "
                             f"no parts for roles {sorted(missing)}; the block's roles are {dict(roles)}")
        parts = {}
        for role, family in roles.items():
            if role not in ls.parts:
                continue
            if family not in PART_FAMILIES:
                raise ValueError(f"block {ls.block!r}: role {role!r} names the unknown family {family!r}")
            parts[role] = PART_FAMILIES[family].build(ls.parts[role].kind, **ls.parts[role].args)
        return block_cls(parts, **dict(ls.block_args))

    def _check_order(self) -> None:
        for n, call in enumerate(self.spec.order):
            src = call.reads_cache_of
            if src is None:
                continue
            mine = {r: m.cache_need() for r, m in self.layers[call.layer].block.mixers().items()}
            theirs = {r: m.cache_need() for r, m in self.layers[self.spec.order[src].layer].block.mixers().items()}
            for role, need in mine.items():
                other = theirs.get(role)
                same = (isinstance(need, PagedNeed) and type(other) is type(need)
                        and {**vars(need), "window": None} == {**vars(other), "window": None})
                if not same:
                    raise ValueError(
                        f"order[{n}] reads the cache of call {src}, whose layout differs: {need} vs {other}")

    # ---- layers whose launches are the same but for their tensors
    MIN_ALIKE = 6      # one layer as it comes, two that are written down, and enough that follow them

    @staticmethod
    def _listable(layer: Layer) -> bool:
        return all(map(launches_alike, (layer.block, *layer.block.parts.values(), *layer.positions.values(),
                                        *(() if layer.position is None else (layer.position,)))))

    def _find_alike(self) -> dict[int, int]:
        """Rows of calls of the order that differ in nothing but their tensors: first call -> the one after the last."""
        def like_next(n: int) -> bool:
            a, b = self.spec.order[n], self.spec.order[n + 1]
            if a.layer == b.layer or self.stream_inputs[n] is not None or self.stream_inputs[n + 1] is not None:
                return False
            if a.reads_cache_of is not None or b.reads_cache_of is not None:
                return False
            one, two = self.layers[a.layer], self.layers[b.layer]
            return {**vars(one.spec), "prefix": None} == {**vars(two.spec), "prefix": None}

        of_layer = list(map(self._listable, self.layers))
        listable = [of_layer[call.layer] for call in self.spec.order]
        rows, n, calls = {}, 0, len(self.spec.order)
        while n < calls:
            end = n + 1
            while listable[n] and end < calls and listable[end] and like_next(end - 1):
                end += 1
            if end - n >= self.MIN_ALIKE:
                rows[n] = end
            n = end
        return rows

    def _place_row(self, n: int) -> "_RowPlaces | None":
        """Where the tensors of the layers of the row that starts at ``n`` lie (attributes of their parts). ``None`` if the layers
        differ in more: in the form of a tensor, in how the tensors lie to one another (a view of another tensor in one
        layer and none in the next), in a plain attribute, or if an attribute is neither (a method put in place of
        the class's, say)."""
        places, form, sizes, watched = [], None, [], []
        for call in range(n, self._rows_of_alike[n]):
            layer = self.layers[self.spec.order[call].layer]
            block, parts = layer.block, layer.block.parts
            if not self._listable(layer):
                return None
            of = [vars(part) for part in parts.values()]
            roles = {id(part): role for role, part in parts.items()}           # (the block's names for its parts)
            own = [roles.get(id(v), v) for v in vars(block).values() if v is not parts]
            values = list(chain(own, *map(dict.values, of)))
            types = list(map(type, values))
            now = [v for v, t in zip(values, types) if t in _TENSORS]
            plain = [v for v, t in zip(values, types) if t in _PLAIN]
            if len(now) < 2 or len(now) + len(plain) != len(values) or any(type(v) in _TENSORS for v in own):
                return None
            at = [t.data_ptr() for t in now]
            starts = [p - t.storage_offset() * t.element_size() for p, t in zip(at, now)]
            first = [starts.index(p) for p in starts]          # the first tensor of the same memory
            mine = (list(parts), list(chain(vars(block), *of)), types, plain, layer.position, layer.positions,
                    [(t.shape, t.dtype, t.stride(), f, p - at[f]) for t, f, p in zip(now, first, at)])
            if form is None:
                form, sizes = mine, [t.numel() * t.element_size() for t in now]
            elif mine != form:
                return None
            watched += [vars(layer), parts, *of, vars(block)]
            places += at
        return _RowPlaces(self.layers, watched, places, sizes)

    def weight_bytes(self, row: int) -> int:
        """The bytes of the tensors of one layer of such a row."""
        return sum(self._row_places[row].sizes)

    def alike_from(self, n: int) -> int:
        """If a row of calls starts at ``n`` whose launches are the same but for their tensors, the call after its last
        one; else 0."""
        return self._rows_of_alike[n] if self._row_places.get(n) is not None else 0

    def places_of_alike(self, row: int, calls: range, caches: list[Any]) -> "tuple[array[int], list[int]] | None":
        """Where the tensors of these calls of the row that starts at ``row`` lie, weights and caches, call by call, and the
        bytes of each of a call's; ``None`` if the layers, since their tensors were bound, or the caches are not alike."""
        if not self._row_places[row].hold():
            self._row_places[row] = self._place_row(row)
            if self._row_places[row] is None:
                return None
        weights, sizes = self._row_places[row].places, self._row_places[row].sizes
        like = [caches[i] for i in self._cache_indices[calls[0]]]
        if any(type(e) is not KVCacheEntry for e in like):
            return None
        form = [(e.group, e.page_size, e.k.shape, e.v.shape) for e in like]
        count, places = len(sizes), []
        for n in calls:
            places += weights[(n - row) * count: (n - row + 1) * count]
            for i, (group, page_size, k_shape, v_shape) in zip(self._cache_indices[n], form):
                e = caches[i]
                if type(e) is not KVCacheEntry or e.group != group or e.page_size != page_size or e.k.shape != k_shape or e.v.shape != v_shape:
                    return None
                places += (e.k.data_ptr(), e.v.data_ptr())
        return array("Q", places), sizes + [t.numel() * t.element_size() for e in like for t in (e.k, e.v)]

    # ---- weights
    def _each_part(self):
        yield "", self.embedding
        for layer in self.layers:
            for part in layer.block.parts.values():
                yield layer.spec.prefix, part
        for part in self.stream_inputs:
            if part is not None:
                yield "", part
        yield "", self.final_norm
        yield "", self.head

    def tensor_specs(self) -> list[TensorSpec]:
        specs: list[TensorSpec] = []
        for prefix, part in self._each_part():
            specs.extend(part.tensor_specs(prefix))
        return list(merge_specs(specs).values())

    def ignorable_tensors(self) -> set[str]:
        out: set[str] = set()
        for prefix, part in self._each_part():
            out |= part.ignorable_tensors(prefix)
        return out

    def bind(self, tensors: Mapping[str, torch.Tensor]) -> None:
        for prefix, part in self._each_part():
            part.bind(prefix, tensors)
        self._row_places = {n: self._place_row(n) for n in self._rows_of_alike}

    # ---- cache
    def cache_needs(self) -> list[CacheNeed | None]:
        """One entry per cache user (a call of the order, a mixer role of its block and a need of
        that mixer; with one mixer per block that keeps one thing, one entry per call): what it keeps
        between steps (``None`` for a mixer that keeps nothing or a call that reads another call's cache)."""
        return list(self._needs)

    def caches_of_call(self, n: int, entries: list[Any]) -> dict[str, Any]:
        """The cache entries that call ``n`` of the order works on, by mixer role: its own, or
        those of the call whose cache it reads."""
        call = self.spec.order[n]
        src = n if call.reads_cache_of is None else call.reads_cache_of
        out = {}
        for role in self.layers[call.layer].block.mixers():
            index = self._user_index[(src, role)]
            entry = tuple(entries[i] for i in index) if isinstance(index, tuple) else entries[index]
            if entry is not None:
                out[role] = entry
        return out

    def recordable(self, kind: str) -> bool:
        """Whether steps of this kind ("decode", "prefill") can be recorded: every part allows it."""
        parts = [part for _, part in self._each_part()] + list(self._positions.values())
        return all(kind in part.recordable for part in parts)


def build_parts(spec: ModelSpec) -> ModelParts:
    return ModelParts(spec)


class DecoderModel:
    """Parts with weights on a device, in one dtype, ready to run steps."""

    def __init__(self, config: ModelConfig, tensors: Mapping[str, torch.Tensor],
                 dtype: torch.dtype, device: torch.device | str) -> None:
        if dtype not in (torch.bfloat16, torch.float32):
            raise ValueError(f"dtype must be bfloat16 or float32, got {dtype}")
        self.config = config
        self.spec = config.to_spec()
        self.parts = build_parts(self.spec)
        self.dtype = dtype
        self.device = torch.device(device)
        self.tensors = dict(tensors)
        self.parts.bind(self.tensors)

    @classmethod
    def from_folder(cls, model_dir: str | Path, dtype: torch.dtype,
                    device: torch.device | str = "cuda") -> "DecoderModel":
        from .config.registry import load_config

        config = load_config(model_dir)
        parts = build_parts(config.to_spec())
        tensors = load_tensors(model_dir, parts.tensor_specs(), dtype, device,
                               ignorable=parts.ignorable_tensors())
        return cls(config, tensors, dtype, device)

    @classmethod
    def from_config(cls, config: ModelConfig, seed: int, dtype: torch.dtype,
                    device: torch.device | str = "cuda") -> "DecoderModel":
        """Random weights made on the device (no folder); see ``weights.random_init``."""
        parts = build_parts(config.to_spec())
        tensors = random_bound_tensors(parts.tensor_specs(), seed, dtype, device)
        return cls(config, tensors, dtype, device)

    @property
    def vocab_size(self) -> int:
        return self.spec.vocab_size

    def cache_needs(self) -> list[CacheNeed | None]:
        return self.parts.cache_needs()

    def weight_bytes(self) -> int:
        seen: set[int] = set()
        total = 0
        for t in self.tensors.values():
            if t.data_ptr() not in seen:
                seen.add(t.data_ptr())
                total += t.numel() * t.element_size()
        return total

    @staticmethod
    def _position_data(encoding: PositionEncoding, ctx: StepContext) -> Any:
        key = encoding.key()
        if key not in ctx.position_tables:
            ctx.position_tables[key] = encoding.prepare(ctx)
        return ctx.position_tables[key]

    def _lists_launches(self, n: int, ctx: StepContext) -> int:
        """If the calls of this step from ``n`` on may be launched from a list, the call after them; else 0: not while the step is
        being recorded (a recording runs what else it has beside the step), nor where each call is checked on the host, nor
        where the products alone keep the device busy for longer than ``LISTED_LAYER_US`` a layer: the host is then ahead of
        it without a list, and what a list takes to make is time that the device waits."""
        if not ops.LAUNCH_LISTS or ctx.recorded or self.device.type != "cuda" or ops.CHECK_INDICES:
            return 0
        end = self.parts.alike_from(n)
        if end and self.parts.weight_bytes(n) * ctx.num_tokens > LISTED_LAYER_US * BYTE_TOKENS_PER_US[self.dtype]:
            return 0
        return end

    def _run_call(self, n: int, stream: ResidualStream, ctx: StepContext, caches: list[Any]) -> None:
        parts, call = self.parts, self.spec.order[n]
        layer = parts.layers[call.layer]
        if parts.stream_inputs[n] is not None:
            parts.stream_inputs[n].forward(stream, ctx)
        if layer.positions:
            tables = {role: self._position_data(p, ctx) for role, p in layer.positions.items()}
        else:
            tables = None if layer.position is None else self._position_data(layer.position, ctx)
        ctx.upcoming_caches = parts.caches_of_call(n + 1, caches) if n + 1 < len(self.spec.order) else {}
        layer.block.forward(stream, ctx, parts.caches_of_call(n, caches), call.reads_cache_of is None, tables)

    def _run_alike(self, n: int, end: int, stream: ResidualStream, ctx: StepContext, caches: list[Any]) -> None:
        """Calls ``n`` to ``end``, which differ in nothing but their tensors: the first as it comes (it may find another
        stream than the rest), the next two written down, one in each half of the arena, and what follows
        launched from those two lists, as long as the arena stayed where it was."""
        self._run_call(n, stream, ctx, caches)
        moves = ctx.arena.moves
        noted, left = [], []
        for m in (n + 1, n + 2):
            with launch_list.Noting() as calls:
                self._run_call(m, stream, ctx, caches)
            noted.append(calls)
            left.append((ctx.arena.frame_state(), stream.state()))
        at = self.parts.places_of_alike(n, range(n + 1, end), caches) if ctx.arena.moves == moves else None
        if at is not None and launch_list.run(noted, *at):
            if (end - n - 3) % 2:           # the last layer worked where the first of the two did
                ctx.arena.resume_frame(left[0][0])       # as far as that one used it: its output still lies there
                stream.set_state(left[0][1])
            return
        for m in range(n + 3, end):
            self._run_call(m, stream, ctx, caches)

    def forward(self, ctx: StepContext, caches: list[Any], want_rows: torch.Tensor | None,
                num_want: int) -> torch.Tensor | None:
        """Run this step's tokens; return float32 logits ``[num_want, vocab]`` at ``want_rows``
        (flat row indices into the step's tokens), or ``None`` if nothing is wanted."""
        parts = self.parts
        stream = ResidualStream(parts.embedding.forward(ctx))
        if parts.keeps_origin:
            stream.origin = parts.embedding.forward(ctx)      # a second copy that no layer adds to
        n, calls = 0, len(self.spec.order)
        while n < calls:
            end = self._lists_launches(n, ctx)
            if end:
                self._run_alike(n, end, stream, ctx, caches)
            else:
                self._run_call(n, stream, ctx, caches)
            n = max(n + 1, end)
        ctx.arena.step_region()
        for join in ctx.at_step_end:
            join()
        ctx.at_step_end.clear()
        if num_want == 0:
            return None
        hn = parts.final_norm.forward_rows(stream, want_rows, num_want, ctx)
        logits = ctx.arena.take_step((num_want, self.spec.vocab_size), torch.float32)
        return parts.head.forward(hn, logits)
