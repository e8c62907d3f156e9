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


@pytest.mark.parametrize("name,body", ALLOCATING, ids=[f"{n}-{i}" for i, (n, _) in enumerate(ALLOCATING)])
def test_tensor_memory_is_allocated_before_later_kernels_may_start(name, body) -> None:
    """An allocation blocks until other CTAs of the SM have freed their columns. A kernel that lets later ones start first
    could find them with the columns it needs, each waiting for the other."""
    alloc = re.search(r"\btmem_alloc(_pair)?\(", body).start()
    known = body.index("__syncthreads()", alloc)            # from here on the CTA has its columns
    triggers = [m.start() for m in re.finditer(r"\bpdl_trigger\(\)", body)]
    assert len(triggers) == 1 and triggers[0] > known
