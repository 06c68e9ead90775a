"""Latent attention with keys and values expanded per head against plain sums in 64 bits."""

import math

import pytest
import torch

from tests.test_attention_packed_gpu import _Ctx

pytestmark = pytest.mark.gpu

# Keys, values and the result are each rounded to 8 bits: 2^-8 / sqrt(3) of a number where a rounding is largest, and a key's
# rounding moves scores of size one, and so weights, by as much; three such roundings add up to 2^-8 as root mean squares.
REL = 2.0 ** -8


class _Steps(_Ctx):
    def __init__(self, lens, starts):
        super().__init__(lens, starts)
        self.start_positions = starts


@pytest.mark.parametrize("heads,dim,rot,rank", [(3, 64, 32, 64), (2, 64, 64, 256), (2, 128, 64, 128), (16, 128, 8, 64), (1, 128, 0, 512)])
@pytest.mark.parametrize("lens,starts,page", [([64], [0], 16), ([65, 1, 130], [0, 200, 63], 8), ([300], [500], 64), ([257], [0], 1)])
@pytest.mark.parametrize("gate,sink", [(True, False), (False, True)])
def test_expanded(heads, dim, rot, rank, lens, starts, page, gate, sink):
    from inference_engine_b200.engine.workspace import Workspace
    from inference_engine_b200.kernels import get_ops

    ops, n, row, g = get_ops(), sum(lens), rank + rot, torch.Generator(device="cuda").manual_seed(heads + rank)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    need = [-(-(a + q) // page) for a, q in zip(starts, lens)]
    order = torch.randperm(sum(need) + 2, generator=torch.Generator().manual_seed(1)).tolist()
    cache = rand(sum(need) + 2, 1, page, row).bfloat16()
    tables, rows = torch.full((len(lens), max(need) + 1), -1, dtype=torch.int32), []
    for i, count in enumerate(need):
        pages, order = order[:count], order[count:]
        tables[i, :count] = torch.tensor(pages)
        rows.append(cache[pages].reshape(-1, row)[: starts[i] + lens[i]].double())
    q = rand(n, heads * (dim + rot)).bfloat16().float()  # (so the stage that rounds the queries changes nothing)
    w_kv = (rand(heads * 2 * dim, rank) * rank ** -0.5).bfloat16()
    pre = rand(n, heads + 3)[:, 2: 2 + heads] if gate else None
    sinks = rand(heads) * 2 if sink else None
    scale, ctx = (dim + rot) ** -0.5, _Steps(lens, starts)
    out = torch.empty(n, heads * dim, dtype=torch.bfloat16, device="cuda")
    ops.latent_expanded(q, w_kv, cache, tables.cuda(), ctx, ctx.positions, None, 0, out, heads=heads, dim=dim, rot_dim=rot, vdim=dim,
                        rank=rank, page_size=page, interleaved=True, scale=scale, gate_pre=pre, sinks=sinks, ws=Workspace("cuda"))
    ops.check_errors()
    want, at = [], 0
    uk, uv = w_kv[: heads * dim].double().view(heads, dim, rank), w_kv[heads * dim:].double().view(heads, dim, rank)
    for c, count, a in zip(rows, lens, starts):
        qq = q[at: at + count].double().view(count, heads, dim + rot)
        at += count
        s = torch.einsum("qhd,hdr,kr->hqk", qq[..., :dim], uk, c[:, :rank]) + torch.einsum("qhd,kd->hqk", qq[..., dim:], c[:, rank:])
        seen = torch.arange(a + count, device="cuda")[None, :] <= torch.arange(a, a + count, device="cuda")[:, None]
        s = (s * scale).masked_fill(~seen, -math.inf)
        if sink:
            s = torch.cat([s, sinks.double()[:, None, None].expand(heads, count, 1)], dim=-1)
        p = torch.softmax(s, dim=-1)[..., : a + count]
        want.append(torch.einsum("hqk,kr,hdr->qhd", p, c[:, :rank], uv))
    want = torch.cat(want)
    if gate:
        want = want * torch.sigmoid(pre.double())[..., None]
    want = want.reshape(n, -1)
    rel = float((out.double() - want).norm() / want.norm())
    assert rel < REL, f"{rel:.2e}"


def test_portions_of_a_growing_context_share_a_workspace():
    """Each portion's context is longer than the last one's: the scratch grows, captured addresses (the workspace's version) stay."""
    from inference_engine_b200.engine.workspace import Workspace
    from inference_engine_b200.kernels import get_ops

    ops, heads, dim, rot, rank, page, g = get_ops(), 2, 64, 32, 64, 16, torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    total, portion = 2000, 400
    cache, tables = rand(total // page, 1, page, rank + rot).bfloat16(), torch.arange(total // page, dtype=torch.int32, device="cuda")[None]
    w_kv, shared, outs = (rand(heads * 2 * dim, rank) * rank ** -0.5).bfloat16(), Workspace("cuda", min_rows=portion), []
    for start in range(0, total, portion):
        q, ctx = rand(portion, heads * (dim + rot)), _Steps([portion], [start])
        for ws in (shared, Workspace("cuda")):
            out = torch.empty(portion, heads * dim, dtype=torch.bfloat16, device="cuda")
            ops.latent_expanded(q, w_kv, cache, tables, ctx, ctx.positions, None, 0, out, heads=heads, dim=dim, rot_dim=rot, vdim=dim,
                                rank=rank, page_size=page, interleaved=True, scale=0.1, gate_pre=None, sinks=None, ws=ws)
            outs.append(out)
        assert torch.equal(outs[-1], outs[-2]) and shared.version == 0
    ops.check_errors()


def test_which_steps_expand():
    """Prompts and long portions do; decoding requests, short portions and captured steps of any lengths do not."""
    from inference_engine_b200.kernels import get_ops

    expands = lambda ctx, **s: get_ops().latent_expands(ctx, **{**dict(heads=16, dim=128, rot_dim=64, vdim=128, rank=512), **s})  # noqa: E731
    assert expands(_Steps([2048], [0])) and expands(_Steps([512], [4096])) and expands(_Steps([700, 900], [0, 100]))
    assert not expands(_Steps([1] * 32, [3000] * 32)) and not expands(_Steps([64], [0]))
    assert not expands(_Steps([128] + [1] * 60, [0] + [8000] * 60))
    assert not expands(_Steps([2048], [0]), dim=96) and not expands(_Steps([2048], [0]), rot_dim=12)
    captured = _Steps([2048], [0])
    captured.bounds = (2048, 4, 4096)
    assert not expands(captured)
