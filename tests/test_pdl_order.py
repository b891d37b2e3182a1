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
    read = [p for p in pointers if re.search(rf"(?<![.\w]){p}\b", head)]
    assert not read, f"{kernel} touches {read} above pdl_wait()"


def test_the_grouped_experts_have_no_loads_that_could_move_above_the_wait():
    """Read-only loads (``__ldg``, or what ``const __restrict__`` makes of a load) are not ordered by the wait: an operand may be the
    launch before's result."""
    text = re.sub(r"//[^\n]*", "", (CSRC_DIR / "qexperts.cu").read_text())
    assert "__ldg" not in text and "__restrict__" not in text and "ld.global.nc" not in text
    for name in ("group_rows_kernel", "weighted_sum_kernel", "route_kernel"):
        head = text[re.search(rf"\n{name}\(", text).end():]
        args, body = head[:head.index("{")], head[head.index("{"):]
        head = body[:body.index("pdl_wait();")]
        read = [p for p in re.findall(r"\*\s*(\w+)", args) if re.search(rf"(?<![.\w]){p}\b", head)]
        assert not read, f"{name} touches {read} above pdl_wait()"
