"""Host-side choices of the kernel wrappers that need no GPU: into how many key ranges decode
attention cuts a request."""

from __future__ import annotations

import pytest
import torch

from tinyserve_b200.kernels import ops


@pytest.mark.parametrize("slots", [148, 444, 592])
def test_key_ranges_fit_the_machine_and_leave_room_for_clusters(slots) -> None:
    for ctas in range(1, slots + 50):
        for most in (1, 2, 5, 16, 64):
            plain = ops.choose_splits(ctas, slots, most)
            inside = ops.choose_splits(ctas, slots, most, cluster=True)
            for s in (plain, inside):
                assert 1 <= s <= max(1, most)
                assert s == 1 or s * ctas <= slots
            assert plain <= 12
            assert inside <= ops.CLUSTER_MAX
            if inside > 1:
                assert inside * ctas <= slots - ops.CLUSTER_ROOM * inside
            if inside > 2:
                assert inside * ctas <= ops.CLUSTER_FILL * slots
            if 2 * ctas > slots:
                assert plain == inside == 1


def test_key_ranges_at_the_measured_batches() -> None:
    # 8 kv heads, three CTAs of the TMA kernel per SM: batch -> ranges that measured best
    for batch, want in [(1, 8), (4, 8), (7, 6), (8, 5), (9, 4), (11, 4), (12, 3), (15, 3), (16, 2), (24, 2), (32, 1), (64, 1)]:
        assert ops.choose_splits(batch * 8, 444, 64, cluster=True) == want
    assert ops.choose_splits(8, 444, 3, cluster=True) == 3          # a short context is cut less


def test_without_cluster_merge_the_old_rule_holds(monkeypatch) -> None:
    monkeypatch.setattr(ops, "CLUSTER_MERGE", False)
    assert ops.choose_splits(64, 444, 64, cluster=True) == ops.choose_splits(64, 444, 64) == 6


def test_which_tiles_the_tcgen05_product_takes() -> None:
    """Pairs of CTAs (256-row tiles) where those fill at least 85 % of the rounds they take on 74 pairs,
    single CTAs (128-row tiles) where only those do on 148 SMs, else the vendor library."""
    # 2,048 rows: qkv of the 0.6B sizes (8 x 16 pair tiles: two rounds, 86 %) and of the 8B sizes
    assert ops.tcgen05_tiles(2048, 4096, 256) == "pairs"
    assert ops.tcgen05_tiles(2048, 6144, 256) == "pairs"
    # gate/up with the activation in the epilogue: tiles of 128 output columns
    assert ops.tcgen05_tiles(2048, 3072, 128) == "pairs"
    # narrow outputs (o and down of the 0.6B sizes: 32 pair tiles) and 320 tiles of 2.2 rounds: the library
    assert ops.tcgen05_tiles(2048, 1024, 256) == ""
    assert ops.tcgen05_tiles(2048, 5120, 256) == ""
    # nine 128-row tiles x sixteen fill 148 SMs (97 %), five 256-row tiles x sixteen do not fill 74 pairs twice
    assert ops.tcgen05_tiles(1152, 2048, 128) == "single"
    assert ops.tcgen05_tiles(2304, 2048, 128) == "pairs"
    for m in (128, 512, 2048, 8192):
        for n in (1024, 4096, 24576, 151936):
            kind = ops.tcgen05_tiles(m, n, 256)
            if kind == "pairs":
                assert ops.tcgen05_pairs_fill_the_machine(m, n, 256)
            elif kind == "single":
                assert ops.tcgen05_fills_the_machine(m, n, 256) and not ops.tcgen05_pairs_fill_the_machine(m, n, 256)
            else:
                assert not ops.tcgen05_fills_the_machine(m, n, 256)


def test_pairs_can_be_switched_off(monkeypatch) -> None:
    monkeypatch.setattr(ops, "TCGEN05_PAIR", False)
    assert ops.tcgen05_tiles(2048, 4096, 256) == "single"


def test_parts_of_the_sums_of_squares_that_the_stream_product_leaves() -> None:
    """``ts_gemm_skinny_to_stream`` cuts narrow outputs into tiles of 8 columns (N / 8 parts of the rows'
    sums of squares) where that spreads the weights better over the SMs and all of K fits a CTA's loads in
    flight, else into tiles of 16; the rule is a host function of the library, so it runs without a GPU.
    The product that folds the norm in adds up at most 128 parts a row."""
    from tinyserve_b200.kernels.build import KernelBuildError, library

    try:
        parts = library().ts_gemm_skinny_to_stream_parts
    except (KernelBuildError, OSError) as e:      # no nvcc or no CUDA runtime on this host
        pytest.skip(f"the kernel library cannot be built or loaded here: {e}")
    assert parts(1, 1024, 2048) == parts(8, 1024, 3072) == parts(16, 1024, 2048) == 128      # o and down of the 0.6B sizes
    assert parts(8, 1024, 4096) == 64                  # K too long for one CTA's loads in flight
    assert parts(8, 2048, 1024) == 128                 # 128 tiles of 16 columns: halves spread no better
    assert parts(8, 4096, 4096) == 256
    for n in range(16, 2049, 16):
        for m in (1, 8, 9, 16):
            p = parts(m, n, 1024)
            assert p in (n // 16, n // 8)
            assert p == n // 16 or p <= 128


def test_one_head_or_two_a_cta_in_the_prompt_attention() -> None:
    """One head where its CTAs all run at once, two where one head's would queue; windows and single tokens count as they run."""
    from types import SimpleNamespace

    def choice(query_lens, context_lens, heads=16, kv_heads=8, window=0):
        return ops._prefill_heads_per_cta(SimpleNamespace(query_lens=query_lens, context_lens=context_lens), heads, kv_heads, window)

    assert choice([512], [512]) == 1 and choice([512], [4096]) == 1
    assert choice([2048], [2048]) == 1 and choice([2048], [9001]) == 2 and choice([8192], [8192]) == 2
    assert choice([290] * 7, [290] * 7) == 2
    assert choice([2048, 1, 1], [9001, 500, 70]) == 2 and choice([1], [100]) == 1
    assert choice([2048], [9001], window=128) == choice([2048], [2176], window=128)
    assert choice([8192], [8192], heads=24) == 1          # three heads a group: no pairs


def test_one_head_or_two_a_cta_by_the_head_size_and_a_recorded_portion_s_note_of_it() -> None:
    """Heads of 64 and of 128 lie on different sides where the two forms were measured to; a step notes which of its layouts have
    which, so that the note alone gives the choice again."""
    from types import SimpleNamespace

    assert ops.prefill_heads_per_cta([1024], [1024], 32, 8) == 1 and ops.prefill_heads_per_cta([1024], [1024], 32, 8, 0, 64) == 2
    for d in (64, 128):
        assert ops.prefill_heads_per_cta([512], [512], 16, 8, 0, d) == 1 and ops.prefill_heads_per_cta([4096], [4096], 16, 8, 0, d) == 2
        ctx = SimpleNamespace(query_lens=[1024], context_lens=[1024], prompt_heads={})
        heads = ops._prefill_heads_per_cta(ctx, 32, 8, 0, d)
        (layout, noted), = ctx.prompt_heads.items()
        assert noted == heads == ops.prefill_heads_per_cta([1024], [1024], *layout)


def test_expert_products_of_a_few_tokens_by_their_ctas_per_k() -> None:
    """On either side of the line, shapes measured on both; never beyond the 16 rows that the form holds."""
    take = ops.moe_takes_few_rows
    for tokens, experts, top, n, k, gated in [(4, 16, 3, 768, 1024, True), (4, 16, 3, 1024, 768, False), (2, 8, 2, 14336, 4096, True),
                                              (8, 8, 2, 4096, 14336, False), (4, 128, 8, 1536, 4096, True), (1, 16, 3, 768, 256, True),
                                              (8, 128, 8, 2048, 768, False), (16, 4, 2, 512, 512, False)]:
        assert take(tokens, experts, top, n, k, gated)
    for tokens, experts, top, n, k, gated in [(8, 8, 2, 14336, 4096, True), (16, 128, 8, 1536, 4096, True), (8, 16, 3, 768, 256, True),
                                              (16, 128, 8, 2048, 768, False), (8, 64, 8, 1024, 384, False), (16, 64, 6, 1408, 2048, True),
                                              (17, 4, 2, 64, 4096, True), (17, 4, 2, 64, 4096, False)]:
        assert not take(tokens, experts, top, n, k, gated)
    assert take(1, 2, 2, 64, 64, True) and not take(1, 2, 2, 1 << 20, 64, True)


def test_few_rows_of_large_matrices_by_the_shape_of_the_matrix() -> None:
    """The tcgen05 kernel of a few rows takes the matrices that it was measured to stream faster than the library, whatever
    kind of product they come from; single products on either side of each line."""
    def take(m, n, k, swiglu=False, dtype=torch.bfloat16):
        def like(*shape):
            return torch.empty(1, dtype=dtype).expand(shape)          # (sizes and types decide: no memory behind it)
        return ops.takes_rows_tcgen05(like(m, k), like(2 * n if swiglu else n, k), like(m, n), swiglu)

    assert take(1, 4096, 4096) and take(16, 6144, 4096) and take(5, 10240, 5120) and take(1, 2048, 8192)
    assert not take(17, 6144, 4096) and not take(1, 10248, 5120) and not take(1, 2040, 16384) and not take(1, 8192, 2560)
    assert not take(1, 4096, 4088) and not take(1, 4096, 4100) and not take(1, 4096, 4096, dtype=torch.float32)
    assert take(1, 12288, 4096, True) and take(16, 1024, 8192, True) and take(1, 16384, 512, True)
    assert not take(1, 512, 16384, True) and not take(1, 32768, 256, True) and not take(17, 12288, 4096, True)


def test_latent_attention_of_single_tokens_by_16_heads_a_cta_or_64() -> None:
    """Shapes measured on both sides (the comment at ``latent_form``): few heads, few requests or few keys take 16 heads a CTA."""
    for requests, heads, keys, rank, d, rows64 in [(1, 16, 4000, 512, 576, False), (64, 32, 4000, 512, 576, False), (1, 64, 60000, 512, 576, False),
                                                   (4, 64, 500, 512, 576, False), (1, 128, 16000, 512, 576, False), (16, 8, 500, 128, 144, False),
                                                   (4, 64, 16000, 512, 576, True), (64, 64, 4000, 512, 576, True), (64, 128, 200, 512, 576, True),
                                                   (256, 128, 2000, 512, 576, True), (16, 64, 4000, 128, 192, True)]:
        form, splits = ops.latent_form(requests, heads, keys, rank, d)
        assert form == rows64, (requests, heads, keys)
        if rows64:
            assert splits == ops.latent_splits_rows64(requests, heads, keys) <= 16 and splits * 64 <= max(64, keys)
        else:
            assert splits == ops.latent_splits(requests, heads, keys) <= 8
    for requests in range(1, 300, 7):
        for heads in (1, 16, 17, 64, 65, 128):
            for keys in (1, 63, 64, 129, 5000):
                form, splits = ops.latent_form(requests, heads, keys, 512, 576)
                assert 1 <= splits <= (16 if form else 8) and splits * requests * -(-heads // (64 if form else 16)) <= max(148, requests * -(-heads // (64 if form else 16)))


def test_mlstm_over_chunks_by_the_step_and_its_scratch() -> None:
    """Steps measured on both sides (the comment at ``mlstm_chunk_heads``): many short portions beside one of 128 go token by token.
    The scratch stays within its limit, whatever the step."""
    def some(lens, heads=8, d=128, dv=128):
        return ops.mlstm_chunk_heads(sum(lens), len(lens), max(lens), heads, d, dv)

    for lens in ([128], [256], [2048], [128] * 16, [800] * 8, [1] * 64 + [400], [100, 370, 650]):
        assert some(lens) == 8
    for lens in ([127], [1] * 64, [1] * 64 + [128], [1] * 256 + [128], [4] * 255 + [150], [100] * 63 + [130]):
        assert some(lens) == 0
    assert some([1] * 64 + [400], heads=16) == 0 and some([256], d=129) == 0
    assert some([1] * 256 + [128], 4, 64, 64) and not some([1] * 256 + [128], 2, 64, 512) and some([1] * 64 + [128], 2, 64, 512)
    for lens in ([2048], [800] * 8, [128] * 64, [8192] * 4, [300000]):
        for heads, d, dv in ((8, 128, 128), (64, 128, 512), (16, 64, 64), (3, 1, 1)):
            n = some(lens, heads, d, dv)
            assert 0 <= n <= heads and 4 * (sum(lens) // 64 + len(lens)) * n * d * dv <= 1 << 26
    assert 0 < some([800] * 8, 64) < 64 and some([1 << 21]) == 0
