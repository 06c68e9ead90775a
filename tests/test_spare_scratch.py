"""Scratch that a faster way through a step takes and another way does without: it grows by doubling, leaves captured steps alone
where none uses it, and stays within what the engine has room for (no GPU needed)."""

from __future__ import annotations

import types

import pytest
import torch

from inference_engine_b200.engine.workspace import Workspace
from inference_engine_b200.kernels.cuda_ops import CudaOps

LATENT = dict(heads=8, dim=64, rot_dim=32, vdim=64, rank=256)


def _ops():
    ops = types.SimpleNamespace(torch=torch, latent_expand=True, EXPANDED_MOST=CudaOps.EXPANDED_MOST, chunks_always=True, CHUNK=CudaOps.CHUNK)
    for name in ("_expanded_wants", "latent_expands", "latent_scratch_bytes", "_recurrence_chunks", "chunk_scratch_bytes"):
        setattr(ops, name, getattr(CudaOps, name).__get__(ops))
    floats = lambda chunks, heads, dim, vdim, delta: chunks * heads * dim * vdim  # noqa: E731
    lib = types.SimpleNamespace(ie_chunked_ok=lambda dim, vdim, delta: dim <= 128, ie_chunked_scratch=floats)
    ops._part_lib = lambda name: lib
    return ops


def _ctx(ws, lens, starts):
    return types.SimpleNamespace(ws=ws, bounds=None, q_lens=lens, start_positions=starts, max_q_len=max(lens))


def test_a_long_prompt_in_portions_leaves_captured_steps_alone():
    """16,384 tokens in portions of 2,048: the expanded keys and values grow with every portion."""
    ops, ws = _ops(), Workspace("cpu", min_rows=2048)
    ws.buffer("hidden", 2048, 8, torch.float32)
    places = set()
    for start in range(0, 16384, 2048):
        ctx = _ctx(ws, [2048], [start])
        assert ops.latent_expands(ctx, **LATENT)
        views = ws.spare(ops._expanded_wants(start + 2048, **LATENT), captured=False)
        assert [tuple(v.shape) for v in views] == [(start + 2048, 288), (start + 2048, 1024)]
        places.add(views[1].data_ptr())
        assert ws.version == 0
    assert len(places) <= 4  # (doubled, not replaced for every portion)


def test_the_chunks_scratch_grows_by_doubling():
    ops, ws = _ops(), Workspace("cpu", min_rows=2048)
    versions = []
    for tokens in range(64, 64 * 33, 64):
        chunks, scratch = ops._recurrence_chunks(_ctx(ws, [tokens], [0]), 2, 16, 16, False, ())
        assert chunks == tokens // 64 and scratch.numel() == chunks * 2 * 16 * 16 and scratch.dtype == torch.float32
        versions.append(ws.version)
    assert versions[-1] == 5 and versions[16:] == [5] * 16  # (captured steps use it: 1 -> 2, 4, 8, 16, 32 chunks)
    assert ws.bytes() == 4 * 32 * 2 * 16 * 16


def test_what_there_is_no_room_for_is_done_without():
    ops, ws = _ops(), Workspace("cpu")
    ctx = _ctx(ws, [2048], [0])
    need = sum(2 * rows * cols for _, rows, cols, _ in ops._expanded_wants(2048, **LATENT))
    ws.spare_bytes = need - 1
    assert not ops.latent_expands(ctx, **LATENT) and ws.spare(ops._expanded_wants(2048, **LATENT)) is None and ws.bytes() == 0
    ws.spare_bytes = need  # (no room to double: exactly what is needed)
    assert ops.latent_expands(ctx, **LATENT)
    assert ws.spare(ops._expanded_wants(2048, **LATENT), captured=False) is not None and ws.bytes() == need
    assert ops._recurrence_chunks(ctx, 2, 16, 16, False, ()) == (0, None)  # (the two kinds together stay within it)
    ws.spare_bytes = need + 4 * 32 * 2 * 16 * 16
    assert ops._recurrence_chunks(ctx, 2, 16, 16, False, ())[0] == 32
    assert not ops.latent_expands(_ctx(ws, [2048], [1]), **LATENT)
    assert ws.bytes() == ws.spare_bytes and ws.version == 0


@pytest.mark.parametrize("utilization,share", [(0.9, 1.0), (0.1, 0.25)])
def test_the_cache_leaves_room_for_it(monkeypatch, utilization, share):
    """What the engine may fill holds the cache and the scratch; of a small room no more than a part in 32 goes to scratch."""
    from inference_engine_b200.cache import storage

    gib, group = 2**30, types.SimpleNamespace(bytes_per_page=lambda page, size: 2**20)
    free = [170 * gib]
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device: (free[0], 180 * gib))
    spare = 2 * gib
    plain = storage.pages_that_fit([group], 16, 2, "cuda", utilization)
    pages = storage.pages_that_fit([group], 16, 2, "cuda", utilization, spare)
    room = utilization * 180 * gib - 10 * gib - storage.HEADROOM_BYTES
    assert plain == int(room // 2**20) and plain - pages == pytest.approx(min(spare, room / 32) / 2**20, abs=1)
    free[0] -= pages * 2**20
    left = storage.spare_that_fits("cuda", utilization)
    assert left == pytest.approx(min(spare, room / 32), abs=2**20) and (left >= spare * 0.999) == (share == 1.0)
    free[0] = 0
    assert storage.spare_that_fits("cuda", utilization) == 0 and storage.spare_that_fits("cpu", utilization) is None


def test_a_model_says_what_it_could_use():
    """Layers of one kind share their scratch; a 32-bit model uses none."""
    from inference_engine_b200.engine.model import Model
    from inference_engine_b200.parts.delta_rule import ChannelDeltaRule
    from inference_engine_b200.parts.latent_attention import LatentAttention

    latent, delta, parts = object.__new__(LatentAttention), object.__new__(ChannelDeltaRule), []
    latent.heads, latent.dim, latent.rot_dim, latent.vdim, latent.kv_rank = 16, 128, 64, 128, 512
    delta.heads, delta.dim, delta.vdim = 16, 128, 128
    ops = _ops()
    ops.takes_chunks = True
    model = types.SimpleNamespace(all_parts=lambda: parts)
    need = lambda tokens, seqs, context: Model.spare_scratch_bytes(model, ops, tokens, seqs, context)  # noqa: E731
    assert need(4096, 64, 10**6) == 0
    for part in (latent, delta):
        part.dtype = torch.bfloat16
    parts += [latent, latent, delta]
    chunks = 4 * (4096 // 64 + 64) * 16 * 128 * 128
    most = CudaOps.EXPANDED_MOST // (16 * 256)
    assert need(4096, 64, 10**9) == chunks + 2 * most * (16 * 256 + 576)
    assert need(4096, 64, 1000) == chunks + 2 * 1000 * (16 * 256 + 576)
    for part in (latent, delta):
        part.dtype = torch.float32
    assert need(4096, 64, 10**9) == 0
