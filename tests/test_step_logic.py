"""The step function, the cache manager and trace replay on the CPU, with the kernels'
plain references in the kernels' place: every way of cutting requests into steps must give
the plain implementation's logits. (The kernels themselves are tested on the GPU.)"""

from __future__ import annotations

from pathlib import Path

import pytest
import torch

import plain_qwen3 as plain
import replay_cases as cases
from kernel_refs import use_references
from tiny_configs import TINIES, random_prompt, write_tiny

from tinyserve_b200.engine.replay import Replayer
from tinyserve_b200.model import DecoderModel

LENGTHS = {"A": [5, 17, 33, 70], "B": [1, 9, 24, 40, 63], "C": [3, 50, 31]}


def _run(model_dir: Path, page: int, steps, max_tokens: int) -> dict[str, dict[int, torch.Tensor]]:
    """Replay ``steps``; returns logits by request id and absolute position."""
    model = DecoderModel.from_folder(model_dir, torch.float32, "cpu")
    rep = Replayer(model, max_tokens, page_size=page)
    got: dict[str, dict[int, torch.Tensor]] = {}
    fed: dict[str, int] = {}
    for entries, end in steps:
        logits = rep.run_step(entries, end)
        row = 0
        for rid, toks, places in entries:
            base = fed.get(rid, 0)
            for p in places:
                got.setdefault(rid, {})[base + p] = logits[row].clone()
                row += 1
            fed[rid] = base + len(toks)
    rep.cache.check_invariant()
    assert all(g.allocator.num_used == 0 for g in rep.cache.groups), "pages leaked"
    return got


@pytest.mark.parametrize("name", sorted(TINIES))
def test_every_cut_gives_the_plain_logits(name: str, tmp_path: Path) -> None:
    cfg, page, seed = TINIES[name]
    folder = write_tiny(tmp_path, name, torch.float32)
    pcfg, pw = plain.read_config(folder), plain.read_weights(folder, torch.float32)
    reqs = {f"r{i}": random_prompt(n, cfg["vocab_size"], 10 * seed + i) for i, n in enumerate(LENGTHS[name])}
    want = {rid: plain.forward(pcfg, pw, toks) for rid, toks in reqs.items()}
    with use_references():
        for rid, toks in reqs.items():
            for steps in (cases.whole(rid, toks), cases.tail_decoded(rid, toks, 32), cases.portions(rid, toks, seed)):
                got = _run(folder, page, steps, cases.max_live_tokens(steps))
                for pos, row in got[rid].items():
                    torch.testing.assert_close(row, want[rid][pos], atol=2e-5, rtol=2e-5)
                assert len(got[rid]) == len(toks)
        steps = cases.mixed(reqs, seed)
        got = _run(folder, page, steps, cases.max_live_tokens(steps))
        for rid, toks in reqs.items():
            assert len(got[rid]) == len(toks)
            for pos, row in got[rid].items():
                torch.testing.assert_close(row, want[rid][pos], atol=2e-5, rtol=2e-5)


def test_a_recorded_portion_replays_the_form_of_its_own_context() -> None:
    """The recording of a prompt portion serves every context up to a limit: it is chosen by the request's own length, not
    by the limit; a choice that was not recorded takes the recording that shares most of it."""
    from tinyserve_b200.engine.step import PrefillGraph

    class Recording:
        def __init__(self, name: str) -> None:
            self.name = name

        def replay(self) -> None:
            replayed.append(self.name)

    replayed: list[str] = []
    g = object.__new__(PrefillGraph)
    g.tokens, g.layouts = 2048, {(16, 8, 0): 2, (16, 16, 0): 1}
    assert g.form_of(2048) == (1, 1) and g.form_of(9001) == (2, 1)
    g.graphs = {(1, 1): Recording("one"), (2, 1): Recording("two")}
    for total in (2048, 9001, 2100, 8192):
        g.replay(total)
    assert replayed == ["one", "two", "one", "two"]
    g.layouts = {(16, 8, 0): 2, (32, 8, 0): 2, (16, 16, 0): 1}
    g.graphs = {(1, 1, 1): Recording("a"), (2, 2, 1): Recording("b")}
    assert g.form_of(2048) == (1, 2, 1)
    g.replay(9001)
    g.replay(2048)
    assert replayed[4] == "b" and replayed[5] in "ab"


def test_an_arena_that_finds_no_memory_asks_for_none_of_it_later(monkeypatch) -> None:
    """Who can do without (the mLSTM's scratch) catches the error and goes on: neither this step's other takes nor the buffer that
    holds the next whole step are to be as large as what failed."""
    from tinyserve_b200.engine import arena as module

    arena, empty = module.Arena("cpu"), torch.empty

    def limited(*shape, **kw):
        if kw.get("dtype") is torch.uint8 and shape[0] > 1 << 20:
            raise torch.cuda.OutOfMemoryError("no memory")
        return empty(*shape, **kw)

    monkeypatch.setattr(module.torch, "empty", limited)
    for _ in range(3):
        arena.begin_step()
        arena.next_frame()
        a = arena.take((1000,), torch.float32)
        with pytest.raises(torch.cuda.OutOfMemoryError):
            arena.take((1 << 21,), torch.uint8)
        b = arena.take((1000,), torch.float32)
        assert a.data_ptr() + 4000 <= b.data_ptr() or b.data_ptr() + 4000 <= a.data_ptr()
    assert arena.reserved_bytes < 1 << 20
