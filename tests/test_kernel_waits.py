"""Every kernel that may be launched while the one before it still runs waits for it on every way out.

`common.cuh`: "my predecessor is done" holds transitively because every thread waits (`ie_pdl_wait`), or, where blocks without work
leave early, the grid's first block does (`ie_pdl_leave`).  A grid whose blocks all left without waiting would be done at once, and the kernel behind it would take that for the end of everything ahead of it: a captured step
whose portions all have few rows launches a prompt attention in which no block has work, behind a decode attention that still
writes the output.  That depends on timing, so it is looked for in the source."""

from __future__ import annotations

import re
from pathlib import Path

import pytest

import inference_engine_b200

SOURCES = sorted((Path(inference_engine_b200.__file__).parent / "csrc").glob("*.cu"))


def _plain(text: str) -> str:
    text = re.sub(r"/\*.*?\*/", " ", text, flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _block(text: str, at: int) -> str:
    """What stands between the first brace from ``at`` on and its partner."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return text[start + 1: i]
    raise ValueError("a brace without a partner")


def _kernels(text: str):
    """(name, body) of every __global__ function."""
    text = _plain(text)
    for match in re.finditer(r"__global__", text):
        brace, semicolon = text.find("{", match.end()), text.find(";", match.end())
        if brace < 0 or 0 <= semicolon < brace:
            continue  # (a declaration)
        head = text[match.end(): brace]
        head = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", " ", head)
        yield re.search(r"(\w+)\s*\(", head).group(1), _block(text, match.end())


def _leaves_unwaited(body: str) -> bool:
    """Whether a way out stands in front of the wait that the other threads come to (`ie_pdl_leave` directly in front of it will do)."""
    body = re.sub(r"\[[&=]?\]\s*\([^()]*\)(?:\s*->\s*\w+)?\s*\{(?:[^{}]|\{[^{}]*\})*\}", "{}", body)  # (functions inside)
    body = re.sub(r"ie_pdl_leave\(\);\s*return;", "", body)
    wait = body.find("ie_pdl_wait()")
    return re.search(r"\breturn\b", body[: wait if wait >= 0 else len(body)]) is not None


@pytest.mark.parametrize("source", SOURCES, ids=lambda p: p.name)
def test_no_way_out_in_front_of_the_wait(source):
    kernels = [(name, body) for name, body in _kernels(source.read_text()) if "ie_pdl_wait" in body or "ie_pdl_trigger" in body]
    for name, body in kernels:
        assert "ie_pdl_wait()" in body, f"{name} starts early and never waits"
        assert not _leaves_unwaited(body), f"{name} leaves in front of its wait"


def test_the_look_itself():
    early = "__global__ void __launch_bounds__(32 * (1 + 2)) k(int* p) { ie_pdl_trigger(); if (!p) return; ie_pdl_wait(); p[0] = 1; }"
    (name, body), = _kernels(early)
    assert name == "k" and _leaves_unwaited(body)
    (_, body), = _kernels(early.replace("if (!p) return;", "if (!p) { ie_pdl_leave(); return; }"))
    assert not _leaves_unwaited(body)
    (_, body), = _kernels(early.replace("if (!p) return;", "auto f = [&](int x) { if (x) { return 1; } return 2; };"))
    assert not _leaves_unwaited(body)
    common = _plain((SOURCES[0].parent / "common.cuh").read_text())
    leave = _block(common, common.index("void ie_pdl_leave()"))
    assert "ie_pdl_wait()" in leave and all(f"blockIdx.{axis} == 0" in leave for axis in "xyz")
    seen = [name for source in SOURCES for name, _ in _kernels(source.read_text())]
    assert {"attention_packed_kernel", "attention_prefill_tc5_kernel", "attention_decode_kernel"} <= set(seen)


@pytest.mark.parametrize("source", SOURCES, ids=lambda p: p.name)
def test_words_between_the_blocks_of_a_cluster_order_what_they_hand_over(source):
    """A relaxed arrival at another block's barrier orders nothing but tensor memory, around which tcgen05's fences stand: directly in front of it one that
    orders what came before.  Copies are told to the barrier that the reader waits at by the copies themselves."""
    text = _plain(source.read_text())
    helpers = re.findall(r"void (\w+)\([^{}]*\{\s*asm volatile\(\"mbarrier\.arrive\.relaxed\.cluster", text)
    assert len(helpers) == text.count("mbarrier.arrive.relaxed")
    for helper in helpers:
        calls = [m.start() for m in re.finditer(rf"\b{helper}\(", text)][1:]
        assert calls
        for at in calls:
            before = re.sub(r"\s+", " ", text[max(at - 200, 0): at])
            assert re.search(r'tcgen05\.fence::before_thread_sync;" ::: "memory"\); __syncwarp\(\); if \(lane == 0\) $', before), (helper, before[-90:])
