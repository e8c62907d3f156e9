"""Rules that the CUDA sources keep and that no run can show: read from the text of the kernels."""

from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tinyserve_b200" / "csrc"


def kernel_bodies(text: str) -> list[str]:
    """The bodies of the ``__global__`` functions of a source, without its line comments."""
    text = re.sub(r"//[^\n]*", "", text)
    bodies = []
    for start in re.finditer(r"__global__", text):
        at = text.index("{", start.start())
        depth, end = 0, at
        for end in range(at, len(text)):
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            if depth == 0:
                break
        bodies.append(text[at: end + 1])
    return bodies


ALLOCATING = [(p.name, body) for p in sorted(CSRC.glob("*.cu*")) for body in kernel_bodies(p.read_text())
              if re.search(r"\btmem_alloc(_pair)?\(", body)]


def test_kernels_that_allocate_tensor_memory_are_found() -> None:
    assert {"attention_prefill_tcgen05.cu", "gemm_rows_tcgen05.cu", "gemm_tcgen05.cu"} <= {name for name, _ in ALLOCATING}
    assert len(ALLOCATING) >= 4


def depth_at(text: str, at: int) -> int:
    return text.count("{", 0, at) - text.count("}", 0, at)


@pytest.mark.parametrize("name,body", ALLOCATING, ids=[f"{n}-{i}" for i, (n, _) in enumerate(ALLOCATING)])
def test_tensor_memory_is_allocated_behind_the_wait_for_earlier_kernels(name, body) -> None:
    """An allocation blocks until other CTAs of the SM have freed their columns. A CTA that held columns while it waits for
    an earlier kernel could keep a CTA of that kernel from its own, each waiting for the other. So on every way to an
    allocation there is a wait, not under a condition of its own, whose block is still open. One kernel allocates first,
    which is safe because it fits no SM beside the others (asserted by the compiler)."""
    if name == "gemm_rows_tcgen05.cu":
        assert "TMEM_WAITING_SMEM" in (CSRC / name).read_text()
        assert all("TMEM_ALONE_SMEM" in (CSRC / other).read_text() for other, _ in ALLOCATING if other != name)
        return
    for alloc in (m.start() for m in re.finditer(r"\btmem_alloc(_pair)?\(", body)):
        waits = [m.start() for m in re.finditer(r"^\s*pdl_wait\(\);", body[:alloc], re.MULTILINE)]
        assert any(min(depth_at(body, i) for i in range(w, alloc + 1)) >= depth_at(body, w) for w in waits)
