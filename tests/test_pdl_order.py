"""Launches that overlap: a kernel reads its operands only after the wait for the launch before it."""

from __future__ import annotations

import re

import pytest

from vllm_metal_b200.metal.build import CSRC_DIR


def _kernels(name: str) -> dict[str, tuple[list[str], str]]:
    """``{kernel: (its pointer arguments, the text between the start of its body and the wait)}``."""
    text = re.sub(r"//[^\n]*", "", (CSRC_DIR / name).read_text())
    found = {}
    for m in re.finditer(r"__global__\s+void\s+__launch_bounds__\(.*?\)\n(\w+)\(([^{]*)\)\s*\{", text):
        body = text[m.end():]
        end = body.index("pdl_wait();")
        found[m.group(1)] = (re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)", m.group(2)), body[:end])
    return found


@pytest.mark.parametrize("kernel", ["norm_rope_cache_kernel", "norm_rope_cache_rows_kernel"])
def test_no_operand_is_read_before_the_wait(kernel):
    pointers, head = _kernels("rope_cache.cu")[kernel]
    assert {"q_norm_w", "k_norm_w", "positions", "slot_mapping"} <= set(pointers)
    read = [p for p in pointers if re.search(rf"\b{p}\b", head)]
    assert not read, f"{kernel} touches {read} above pdl_wait()"
