"""Steps whose layers are launched from lists against the same steps launched call by call: the same bits."""

from __future__ import annotations

import pytest
import torch

from tiny_configs import REAL_0_6B, TINY_A, TINY_B, random_prompt

pytestmark = pytest.mark.gpu

SIZES = {"tiny": {**TINY_A, "num_hidden_layers": 9}, "odd": {**TINY_B, "num_hidden_layers": 8},
         "wide": {**REAL_0_6B, "num_hidden_layers": 7, "vocab_size": 2048}}


def logits_of(model, listed: bool, steps, tokens):
    """(logits, launches) of the steps on a cache and an arena of their own, layers from lists or not."""
    from tinyserve_b200.engine.replay import Replayer
    from tinyserve_b200.kernels import ops

    rep = Replayer(model, tokens, page_size=16)
    for g in rep.cache.groups:
        g.kv.fill_(float("nan"))
    before, ops.LAUNCH_LISTS = ops.LAUNCH_LISTS, listed
    start = ops.launch_count
    try:
        out = [rep.run_step(entries, []).float().cpu() for entries in steps]
    finally:
        ops.LAUNCH_LISTS = before
    ops.check_device_errors()
    return torch.cat(out), ops.launch_count - start


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("size", list(SIZES))
def test_layers_from_lists_give_the_same_bits(size, dtype, monkeypatch) -> None:
    """Prompts and single tokens, alone and mixed, few rows and many, on an arena that still grows and on one that does
    not; an even and an odd number of layers, of which the first three run call by call."""
    from tinyserve_b200.config import config_from_dict
    from tinyserve_b200.kernels import launch_list
    from tinyserve_b200.model import DecoderModel

    cfg = SIZES[size]
    model = DecoderModel.from_config(config_from_dict(cfg), 3, dtype, "cuda")
    a, b, c = (random_prompt(n, cfg["vocab_size"], 7 + n) for n in (300, 70, 24))
    steps = [[("b", b[:20], [0, 19])], [("a", a[:200], [199]), ("b", b[20:21], [0])], [("a", a[200:298], [0, 97]), ("b", b[21:60], [38]), ("c", c[:1], [0])],
             [("a", a[298:299], [0]), ("b", b[60:61], [0]), ("c", c[1:2], [0])], [("c", c[2:24], [21])],
             [("a", a[299:], [0])]]
    ran = []
    run = launch_list.run
    monkeypatch.setattr(launch_list, "run", lambda *args: ran.append(run(*args)) or ran[-1])
    want, launches = logits_of(model, False, steps, 512)
    assert not ran
    got, listed = logits_of(model, True, steps, 512)
    assert sum(ran) >= 3 and not want.isnan().any()      # (not while the arena grew)
    assert torch.equal(got, want) and listed == launches


def test_a_layer_off_the_16_byte_grid_is_not_listed(monkeypatch) -> None:
    """The kernels choose their accesses by how the weights lie: such a layer is launched call by call."""
    from tinyserve_b200.config import config_from_dict
    from tinyserve_b200.kernels import launch_list
    from tinyserve_b200.model import DecoderModel

    model = DecoderModel.from_config(config_from_dict(SIZES["tiny"]), 3, torch.float32, "cuda")
    steps = [[("a", random_prompt(50, 256, 1), [49])]]
    name = next(n for n in model.tensors if "layers.5" in n and n.endswith("o_proj.weight"))
    w = model.tensors[name]
    base = torch.empty(w.numel() + 1, device="cuda")
    base[1:].copy_(w.flatten())
    model.tensors[name] = base[1:].view(w.shape)
    model.parts.bind(model.tensors)
    ran = []
    run = launch_list.run
    monkeypatch.setattr(launch_list, "run", lambda *args: ran.append(run(*args)) or ran[-1])
    for _ in range(2):
        want, _ = logits_of(model, False, steps, 64)
        got, _ = logits_of(model, True, steps, 64)
        assert not any(ran) and torch.equal(got, want)


def test_a_tensor_replaced_without_bind_is_followed(monkeypatch) -> None:
    """Another storage under a tensor of a layer behind the third, and another tensor: the listed step reads them."""
    from tinyserve_b200.config import config_from_dict
    from tinyserve_b200.kernels import launch_list
    from tinyserve_b200.model import DecoderModel

    model = DecoderModel.from_config(config_from_dict(SIZES["tiny"]), 3, torch.float32, "cuda")
    prompt = random_prompt(50, 256, 1)
    steps = [[("a", prompt[:40], [39])], [("a", prompt[40:], [9])], [("b", prompt[:30], [29])]]
    ran = []
    run = launch_list.run
    monkeypatch.setattr(launch_list, "run", lambda *args: ran.append(run(*args)) or ran[-1])
    before, _ = logits_of(model, True, steps, 128)
    mixer, mlp = (model.parts.layers[6].block.parts[role] for role in ("mixer", "feed_forward"))
    mixer.w_o.data = mixer.w_o.data * 1.5
    for change in ("storage", "tensor"):
        want, _ = logits_of(model, False, steps, 128)
        ran.clear()
        got, _ = logits_of(model, True, steps, 128)
        assert any(ran) and torch.equal(got, want) and not torch.equal(got, before)
        mlp.w_down = mlp.w_down * 0.5
        before = got


@pytest.mark.parametrize("how", ["flag", "mode"])
def test_library_products_follow_what_torch_is_asked_for(how, monkeypatch) -> None:
    """Products of 30 rows go to the vendor library: with sums in 32 bits asked for, or a mode that sees torch's operations, all
    layers are launched call by call, and the mode sees a product in every layer."""
    from torch.utils._python_dispatch import TorchDispatchMode

    from tinyserve_b200.config import config_from_dict
    from tinyserve_b200.kernels import launch_list
    from tinyserve_b200.model import DecoderModel

    seen = []

    class Sees(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    model = DecoderModel.from_config(config_from_dict(SIZES["wide"]), 3, torch.bfloat16, "cuda")
    steps = [[("a", random_prompt(30, 2048, 1), [29])], [("b", random_prompt(30, 2048, 2), [29])]]
    ran = []
    run = launch_list.run
    monkeypatch.setattr(launch_list, "run", lambda *args: ran.append(run(*args)) or ran[-1])
    matmul = torch.backends.cuda.matmul
    logits_of(model, True, steps, 128)
    assert any(ran)
    ran.clear()
    try:
        if how == "flag":
            matmul.allow_bf16_reduced_precision_reduction = False
            want, _ = logits_of(model, False, steps, 128)
            got, _ = logits_of(model, True, steps, 128)
            assert torch.equal(got, want)
        else:
            with Sees():
                logits_of(model, True, steps, 128)
            products = sum("mm" in name for name in seen)
            assert products >= 2 * SIZES["wide"]["num_hidden_layers"]
    finally:
        matmul.allow_bf16_reduced_precision_reduction = True
    assert ran and not any(ran)
