"""Which layers may be launched from lists (``kernels.launch_list``), and that the library and the Python side agree on
the arguments of the entry points that lists may name. Needs no GPU."""

from __future__ import annotations

import ctypes

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
