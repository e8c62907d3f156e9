"""Which layers may be launched from lists (``kernels.launch_list``), and that the library and the Python side agree on
the arguments of the entry points that lists may name. Needs no GPU."""

from __future__ import annotations

import ctypes
import types

import pytest

from tinyserve_b200.config import config_from_dict
from tinyserve_b200.kernels import build, launch_list, ops
from tinyserve_b200.model import ModelParts
from tiny_configs import TINY_A, TINY_B

LISTED = ["ts_add_rms_norm", "ts_qk_norm_rope_write", "ts_silu_mul", "ts_paged_attention_simt", "ts_prefill_attention_tcgen05",
          "ts_prefill_attention_tma", "ts_prefill_attention_mma", "ts_decode_attention_tma", "ts_decode_attention_tma_fused",
          "ts_decode_attention_mma", "ts_gemm_f32", "ts_gemm_simt", "ts_gemm_rows_tcgen05", "ts_gemm_skinny", "ts_gemm_skinny_swiglu",
          "ts_gemm_skinny_normed", "ts_gemm_skinny_to_stream", "ts_gemm_tcgen05", "ts_gemm_tcgen05_swiglu", "ts_library_gemm"]


@pytest.mark.parametrize("name", LISTED)
def test_the_library_and_the_signatures_agree(name) -> None:
    lib = build.library()
    lib.ts_list_entry.argtypes, lib.ts_list_entry.restype = [ctypes.c_char_p, ctypes.c_void_p, ctypes.c_void_p], ctypes.c_int
    kinds = ctypes.create_string_buffer(65)
    count = ctypes.c_int()
    assert lib.ts_list_entry(name.encode(), ctypes.addressof(count), ctypes.addressof(kinds)) >= 0
    of = {ctypes.c_void_p: b"p", ctypes.c_int: b"i", ctypes.c_longlong: b"l", ctypes.c_float: b"f", ctypes.c_double: b"d"}
    assert kinds.value == b"".join(of[t] for t in ops._SIGNATURES[name])
    assert count.value == len(kinds.value) and launch_list._entry(name) is not None


def test_an_entry_point_that_lists_may_not_name() -> None:
    assert launch_list._entry("ts_embed") is None


def rows_of(config: dict) -> dict[int, int]:
    return ModelParts(config_from_dict(config).to_spec())._rows_of_alike


def test_rows_of_alike_layers() -> None:
    assert rows_of({**TINY_A, "num_hidden_layers": 9}) == {0: 9}
    assert rows_of({**TINY_A, "num_hidden_layers": 6}) == {0: 6}
    assert rows_of({**TINY_B, "num_hidden_layers": 5}) == {}          # too few to be worth it


def test_a_part_that_does_not_say_so_is_launched_as_always() -> None:
    from guzovik_cases import CONFIG_A

    assert rows_of(CONFIG_A) == {}


def with_kinds(config: dict, **kinds: str):
    """The config's spec with other registered kinds in some roles; ``block`` and ``position`` name the layer's own."""
    import dataclasses

    from tinyserve_b200.config import PartSpec

    spec = config_from_dict(config).to_spec()
    layers = []
    for layer in spec.layers:
        parts = {role: PartSpec(kinds.get(role, p.kind), p.args) for role, p in layer.parts.items()}
        layers.append(dataclasses.replace(layer, parts=parts, block=kinds.get("block", layer.block),
                                          position=PartSpec(kinds.get("position", layer.position.kind), layer.position.args)))
    return dataclasses.replace(spec, layers=tuple(layers))


def test_a_derived_class_is_launched_as_always_unless_it_says_so_itself() -> None:
    """A part, a block or a position encoding derived from one that may be listed does something of its own beside what it
    inherits (here an operation that is no launch of the library), so nothing is taken for granted of it."""
    from tinyserve_b200.parts import attention, base, block, mlp, norm, rope

    class HalvedSwiGLU(mlp.SwiGLU):
        def forward(self, x, ctx, stream=None):
            return super().forward(x, ctx, stream=None) * 0.5

    class SameSwiGLU(mlp.SwiGLU):
        same_launches = True

    derived = {
        "feed_forward": (base.FEED_FORWARDS, HalvedSwiGLU), "mixer": (base.MIXERS, type("M", (attention.GQAAttention,), {})),
        "mixer_norm": (base.NORMS, type("N", (norm.RMSNorm,), {})), "block": (base.BLOCKS, type("B", (block.PreNormBlock,), {})),
        "position": (base.POSITION_ENCODINGS, type("R", (rope.RotaryEncoding,), {}))}
    config = {**TINY_A, "num_hidden_layers": 9}
    for role, (family, cls) in derived.items():
        family.register(f"derived_{role}_of_this_test", cls)
        assert ModelParts(with_kinds(config, **{role: f"derived_{role}_of_this_test"}))._rows_of_alike == {}
    base.FEED_FORWARDS.register("same_swiglu_of_this_test", SameSwiGLU)
    assert ModelParts(with_kinds(config, feed_forward="same_swiglu_of_this_test"))._rows_of_alike == {0: 9}
    assert ModelParts(with_kinds(config))._rows_of_alike == {0: 9}


@pytest.mark.parametrize("layers", [6, 7, 8, 9])
@pytest.mark.parametrize("hidden, inner", [(64, 16), (64, 200)])
def test_the_arena_behind_a_list_stands_as_behind_the_layers(layers, hidden, inner, monkeypatch) -> None:
    """Behind an even and an odd number of listed layers: what the last one left pending lies where it would, and so does
    what a stream input takes before the next block turns to the other half, without an overlap of the two."""
    import torch

    from tinyserve_b200.engine.arena import Arena
    from tinyserve_b200.model import DecoderModel
    from tinyserve_b200.parts.base import ResidualStream

    class Model:
        """Layers without a feed-forward: a norm's output, two of a mixer's inner rows and its output, left pending."""

        parts = types.SimpleNamespace(places_of_alike=lambda *a: ())
        _run_alike = DecoderModel._run_alike

        def _run_call(self, n, stream, ctx, caches):
            ctx.arena.next_frame()
            for width in (hidden, inner, inner):
                ctx.arena.take((5, width), torch.bfloat16)
            stream.delta = ctx.arena.take((5, hidden), torch.bfloat16)

    def run(listed: bool):
        stream, ctx, model = ResidualStream(torch.zeros(5, hidden)), types.SimpleNamespace(arena=arena), Model()
        arena.begin_step()
        monkeypatch.setattr(launch_list, "run", lambda noted, *at: listed)
        model._run_alike(0, layers, stream, ctx, [])
        beside = arena.take((5, 2 * hidden), torch.bfloat16)
        return [(t.data_ptr(), t.data_ptr() + t.numel() * t.element_size()) for t in (stream.delta, beside)]

    arena = Arena("cpu")
    for _ in range(3):
        want = run(False)
    got = run(True)
    assert got == want
    (a, b), (c, d) = got
    assert b <= c or d <= a


def test_what_is_put_in_place_of_a_layer_s_tensors_or_attributes_is_seen() -> None:
    """Another storage under a bound tensor, another tensor, a plain attribute, a method or a part of one layer, each
    without ``bind``: the list follows where the layers are still alike, and there is none where they are not."""
    import numpy
    import torch

    from tinyserve_b200.model import DecoderModel
    from tinyserve_b200.parts.base import KVCacheEntry

    def fresh():
        model = DecoderModel.from_config(config_from_dict({**TINY_A, "num_hidden_layers": 9}), 3, torch.float32, "cpu")
        parts = [layer.block.parts for layer in model.parts.layers]
        return model.parts, parts, [layer.block for layer in model.parts.layers]

    def places(of):
        caches = [KVCacheEntry(k=torch.zeros(2, 2, 4, 16), v=torch.zeros(2, 2, 4, 16), page_size=4, group=0) for _ in range(9)]
        got = of.places_of_alike(0, range(1, 9), caches)
        return None if got is None else list(got[0])

    model, parts, _ = fresh()
    names = [v.data_ptr() for part in parts[5].values() for v in vars(part).values() if isinstance(v, torch.Tensor)]
    assert set(names) <= set(places(model))
    down = parts[5]["feed_forward"].w_down
    down.data = down.data.clone()                                     # another storage
    assert down.data_ptr() not in names and down.data_ptr() in places(model)
    old = down.data_ptr()
    parts[5]["feed_forward"].w_down = down.clone()                    # another tensor; the old one may have gone
    del down
    assert parts[5]["feed_forward"].w_down.data_ptr() in places(model) and old not in places(model)
    parts[5]["feed_forward"].w_down = parts[5]["feed_forward"].w_down.double()
    assert places(model) is None and model.alike_from(0) == 0         # another form
    for change in (lambda p, b: setattr(p["mixer"], "scale", 0.5), lambda p, b: setattr(p["mixer"], "forward", lambda *a: None),
                   lambda p, b: setattr(p["feed_forward_norm"], "eps", 0.1), lambda p, b: setattr(b, "feed_forward", p["mixer"]),
                   lambda p, b: setattr(p["mixer"], "q_norm_w", None), lambda p, b: setattr(p["mixer"], "extra", torch.zeros(2)),
                   lambda p, b: setattr(b, "scale_b", torch.ones(3)), lambda p, b: setattr(p["mixer"], "scale", numpy.ones(3)),
                   lambda p, b: vars(p["feed_forward"]).pop("w_down"), lambda p, b: setattr(b, "forward", lambda *a: None)):
        for which in ([5], range(9)):
            model, parts, blocks = fresh()
            assert model.alike_from(0) == 9 and places(model) is not None
            for n in which:
                change(parts[n], blocks[n])
            if len(which) == 1 or isinstance(parts[5]["mixer"].scale, numpy.ndarray) or "forward" in {**vars(parts[5]["mixer"]), **vars(blocks[5])}:
                assert places(model) is None and model.alike_from(0) == 0
    model, parts, blocks = fresh()
    model.layers[4] = model.layers[5]
    got, each = places(model), len(names) + 2
    assert got[3 * each: 3 * each + len(names)] == got[4 * each: 4 * each + len(names)]


def test_a_copy_of_the_layers_looks_for_its_own_tensors() -> None:
    import copy
    import pickle

    import torch

    from tinyserve_b200.model import DecoderModel
    from tinyserve_b200.parts.base import KVCacheEntry

    model = DecoderModel.from_config(config_from_dict({**TINY_A, "num_hidden_layers": 9}), 3, torch.float32, "cpu").parts
    caches = [KVCacheEntry(k=torch.zeros(2, 2, 4, 16), v=torch.zeros(2, 2, 4, 16), page_size=4, group=0) for _ in range(9)]
    for other in (copy.deepcopy(model), pickle.loads(pickle.dumps(model))):
        got, _ = other.places_of_alike(0, range(1, 9), caches)
        assert other.alike_from(0) == 9 and other.weight_bytes(0) == model.weight_bytes(0)
        assert other.layers[7].block.parts["mixer"].w_o.data_ptr() in got and model.layers[7].block.parts["mixer"].w_o.data_ptr() not in got


def test_a_library_product_that_torch_was_asked_to_make_otherwise_is_in_no_list(monkeypatch) -> None:
    """The flag for sums in 32 bits, another library, its tuning, a mode that sees torch's operations, or a library that is not
    where torch's build says: the noted call is one that no list may name."""
    import torch

    monkeypatch.setattr(torch.cuda, "current_blas_handle", lambda: 7)
    note = lambda: ops._library_gemm_call(16, 32, 48, 20, 64, 128, 1)
    assert note() == ("ts_library_gemm", (16, 32, 48, 20, 64, 128, 1, ops._library_gemm_function(), 7)) and launch_list._entry(note()[0])
    matmul = torch.backends.cuda.matmul
    matmul.allow_bf16_reduced_precision_reduction = False
    try:
        assert launch_list._entry(note()[0]) is None
    finally:
        matmul.allow_bf16_reduced_precision_reduction = True
    with monkeypatch.context() as m:
        m.setattr(torch.backends.cuda, "preferred_blas_library", lambda: types.SimpleNamespace(name="Cublaslt"))
        assert launch_list._entry(note()[0]) is None
    with monkeypatch.context() as m:
        m.setattr(torch.cuda.tunable, "is_enabled", lambda: True)
        assert launch_list._entry(note()[0]) is None

    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Sees(TorchDispatchMode):
        def __torch_dispatch__(self, func, types_, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class SeesToo(TorchFunctionMode):
        def __torch_function__(self, func, types_, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    for mode in (Sees, SeesToo):
        with mode():
            assert launch_list._entry(note()[0]) is None
    assert launch_list._entry(note()[0]) is not None
    ops._library_gemm_function.cache_clear()
    try:
        with monkeypatch.context() as m:
            m.setattr(torch.version, "cuda", "99.0")
            assert ops._library_gemm_function() == 0 and launch_list._entry(note()[0]) is None
    finally:
        ops._library_gemm_function.cache_clear()


def test_a_part_that_is_a_torch_module_as_well_keeps_its_parameters() -> None:
    """Parts count what is set on them and leave the setting to the other classes that they are of."""
    import torch

    from tinyserve_b200.parts import FeedForward
    from tinyserve_b200.parts.base import Watched

    class Module(FeedForward, torch.nn.Module):
        def __init__(self):
            torch.nn.Module.__init__(self)
            self.weight = torch.nn.Parameter(torch.zeros(3))

    before = Watched.changes()
    part = Module()
    assert [name for name, _ in part.named_parameters()] == ["weight"] and Watched.changes() > before
    before = Watched.changes()
    del part.weight
    assert not list(part.parameters()) and Watched.changes() == before + 1
