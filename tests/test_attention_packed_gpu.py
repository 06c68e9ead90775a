"""The tcgen05 softmax attention of prompt portions against plain sums in 64 bits: edges of its tiles, every option."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu

# Queries, keys and values are exact and a weight keeps 16 bits of mantissa, so what is left is the result's rounding to 8 bits: at most
# 2^-8 of a number, 2^-8 / sqrt(3) = 2.3e-3 as a root mean square where it is largest.
REL = 2.0 ** -8 / math.sqrt(3.0)


class _Ctx:
    bounds = None

    def __init__(self, lens, starts):
        at = [sum(lens[:i]) for i in range(len(lens) + 1)]
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
        self.q_lens, self.q_starts, self.num_seqs, self.max_q_len, self.num_tokens = lens, at[:-1], len(lens), max(lens), at[-1]
        self.cu_q, self.ctx_lens = i32(at), i32([a + n for a, n in zip(starts, lens)])
        self.seq_of_token = i32([i for i, n in enumerate(lens) for _ in range(n)])
        self.positions = i32([a + j for a, n in zip(starts, lens) for j in range(n)])


def _case(lens, starts, heads, kv_heads, dim, vdim, page, window, keep, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    need = [-(-(a + n) // page) for a, n in zip(starts, lens)]
    order = torch.randperm(sum(need) + 3, generator=torch.Generator().manual_seed(seed)).tolist()
    k, v = rand(sum(need) + 3, kv_heads, page, dim).bfloat16(), rand(sum(need) + 3, kv_heads, page, vdim).bfloat16()
    width = max(need) + 2
    tables, rows = torch.full((len(lens), width), -1, dtype=torch.int32), []
    for i, n in enumerate(need):
        pages, order = order[:n], order[n:]
        tables[i, :n] = torch.tensor(pages)
        rows.append((k[pages].transpose(1, 2).reshape(-1, kv_heads, dim), v[pages].transpose(1, 2).reshape(-1, kv_heads, vdim)))
        if window is not None:  # pages behind every query's window, and past the kept first positions, were given back
            gone = [p for p in range(n) if (p + 1) * page <= starts[i] - window + 1 and p * page >= keep]
            tables[i, gone] = -1
    return rand(sum(lens), heads, dim).bfloat16(), k, v, tables.cuda(), rows


def _want(q, rows, lens, starts, scale, window, keep, softcap, sinks, gate):
    heads, out, at = q.shape[1], [], 0
    for (k, v), n, a in zip(rows, lens, starts):
        group = heads // k.shape[1]
        kk, vv = (t[: a + n].double().repeat_interleave(group, 1) for t in (k, v))
        s = torch.einsum("qhd,khd->hqk", q[at: at + n].double(), kk) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        pos, key = torch.arange(a, a + n, device="cuda")[:, None], torch.arange(a + n, device="cuda")[None, :]
        seen = key <= pos
        if window is not None:
            seen &= (key > pos - window) | (key < keep)
        s = s.masked_fill(~seen, -math.inf)
        if sinks is not None:
            s = torch.cat([s, sinks.double()[:, None, None].expand(heads, n, 1)], dim=-1)
        p = torch.softmax(s, dim=-1)[..., : a + n]
        out.append(torch.einsum("hqk,khd->qhd", p, vv))
        at += n
    out = torch.cat(out)
    if gate is not None:
        out = out * torch.sigmoid(gate.double().view(q.shape[0], heads, -1))
    return out


def _check(lens, starts, heads=4, kv_heads=2, dim=64, page=16, window=None, keep=0, softcap=None, sink=True, gate="head", seed=1):
    from inference_engine_b200.kernels import get_ops

    ops, vdim = get_ops(), dim
    q, k, v, tables, rows = _case(lens, starts, heads, kv_heads, dim, vdim, page, window, keep, seed)
    n, g = q.shape[0], torch.Generator(device="cuda").manual_seed(seed + 50)
    sinks = torch.randn(heads, generator=g, device="cuda") * 2 if sink else None
    cols = {"head": heads, "value": heads * vdim, None: 0}[gate]
    gates = torch.randn(n, cols + 3, generator=g, device="cuda")[:, 1: 1 + cols] if gate else None
    out = torch.full((n, heads * vdim + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    before = ops.launch_counts.get("sink_attention_packed", 0)
    ops.sink_attention(q.view(n, -1), k, v, tables, _Ctx(lens, starts), heads, kv_heads, dim, vdim, page, dim ** -0.5, window, sinks,
                       gates, out[:, : heads * vdim], softcap=softcap, keep_first=keep)
    ops.check_errors()
    assert ops.launch_counts.get("sink_attention_packed", 0) == before + 1
    assert bool((out[:, heads * vdim:] == 7.0).all())
    want = _want(q, rows, lens, starts, dim ** -0.5, window, keep, softcap, sinks, gates).view(n, -1)
    got = out[:, : heads * vdim].double()
    assert torch.isfinite(got).all()
    rel = float((got - want).norm() / want.norm())
    assert rel < REL, f"{rel:.2e}"
    worst = float(((got - want).norm(dim=1) / want.norm(dim=1).clamp(min=1e-30)).max())
    assert worst < 2.0 ** -8 * 1.1, f"a row is {worst:.2e} off"  # (every number at its worst, and a tenth for exponentials and sums)


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("heads,kv_heads", [(2, 2), (4, 1), (6, 2), (8, 1)])
@pytest.mark.parametrize("lens,starts", [([64], [0]), ([127], [0]), ([128], [0]), ([129, 65], [0, 63]), ([257, 1, 300], [0, 500, 129]),
                                         ([700], [1000])])
def test_rows_and_keys(dim, heads, kv_heads, lens, starts):
    _check(lens, starts, heads, kv_heads, dim)


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("window,keep", [(1, 0), (100, 0), (128, 0), (129, 4), (300, 200), (64, 1)])
@pytest.mark.parametrize("lens,starts", [([300], [0]), ([200, 90], [700, 1])])
def test_windows(dim, window, keep, lens, starts):
    _check(lens, starts, dim=dim, window=window, keep=keep)


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("softcap,sink,gate,page", [(None, False, None, 16), (5.0, True, "head", 8), (30.0, False, "value", 64),
                                                    (None, True, "value", 128), (2.0, True, None, 1)])
def test_options(dim, softcap, sink, gate, page):
    _check([200, 70], [0, 333], dim=dim, softcap=softcap, sink=sink, gate=gate, page=page, window=150 if page == 8 else None)


def test_scores_that_grow_along_the_keys():
    """Every tile raises every row's maximum far beyond what the weights may lag behind it."""
    from inference_engine_b200.kernels import get_ops

    ops, n, heads, dim = get_ops(), 600, 2, 128
    q, k, v, tables, rows = _case([n], [0], heads, 1, dim, dim, 16, None, 0, 3)
    q = q.abs() + 0.5
    ramp = torch.arange(n, device="cuda").float() / n
    (kk, vv), = rows
    kk = (kk[:n].float().abs() * 0.05 + ramp[:, None, None] * 0.8).bfloat16()
    pad = torch.zeros(tables.shape[1] * 16, 1, dim, dtype=torch.bfloat16, device="cuda")
    pad[:n] = kk
    pages = tables[0, : -(-n // 16)].long()
    k[pages] = pad.view(-1, 16, 1, dim).transpose(1, 2)[: len(pages)]
    out = torch.empty(n, heads * dim, dtype=torch.bfloat16, device="cuda")
    ops.sink_attention(q.view(n, -1), k, v, tables, _Ctx([n], [0]), heads, 1, dim, dim, 16, 1.0, None, None, None, out)
    want = _want(q, [(kk, vv)], [n], [0], 1.0, None, 0, None, None, None).view(n, -1)
    assert float((out.double() - want).norm() / want.norm()) < REL


@pytest.mark.parametrize("dim,heads,kv_heads", [(64, 6, 2), (64, 2, 2), (128, 8, 1), (128, 4, 2)])
@pytest.mark.parametrize("lens,starts", [([17], [0]), ([129, 1, 65], [0, 500, 63]), ([40, 300], [1500, 129]), ([700], [0])])
@pytest.mark.parametrize("window,page", [(0, 16), (100, 8), (1, 1), (0, 64)])
@pytest.mark.parametrize("shares", [1, 2, 3, 8])
def test_prompt_portions_and_shared_keys(monkeypatch, dim, heads, kv_heads, lens, starts, window, page, shares):
    """Plain attention: all portions in one launch, key tiles cut among the blocks of a cluster (some parts empty).  A weight and a
    result are each rounded by 2^-9 at most, which is 2^-8 in all and, where values cancel in a row, twice that."""
    from inference_engine_b200.kernels import get_ops

    ops = get_ops()
    q, k, v, tables, rows = _case(lens, starts, heads, kv_heads, dim, dim, page, window or None, 0, dim + page)
    ctx, n = _Ctx(lens, starts), q.shape[0]
    ctx.start_positions, ctx.max_ctx_len = starts, max(a + b for a, b in zip(lens, starts))
    monkeypatch.setattr(ops, "prompt_packs", lambda *_: True)
    monkeypatch.setattr(ops, "prompt_shares", lambda *_: shares)
    out, before = torch.full((n, heads * dim), 7.0, dtype=torch.bfloat16, device="cuda"), ops.launch_counts.get("attention_prefill_packed", 0)
    ops.paged_attention(q.view(n, -1), k, v, tables, ctx, heads, kv_heads, dim, page, dim ** -0.5, window, out)
    ops.check_errors()
    assert ops.launch_counts.get("attention_prefill_packed", 0) == before + 1
    want, got = _want(q, rows, lens, starts, dim ** -0.5, window or None, 0, None, None, None).view(n, -1), out.double()
    assert float((got - want).norm() / want.norm()) < 2.0 ** -8
    assert float(((got - want).norm(dim=1) / want.norm(dim=1)).max()) < 2.0 ** -7


def test_a_fixed_launch_serves_shorter_steps():
    """Bounds for 256 tokens of 4 requests over 2,048 positions, a step of less: blocks without rows leave, parts may be empty."""
    from inference_engine_b200.kernels import get_ops

    ops, lens, starts = get_ops(), [100, 1, 20], [30, 700, 0]
    for dim in (64, 128):
        q, k, v, tables, rows = _case(lens, starts, 8, 2, dim, dim, 16, None, 0, dim)
        ctx, n = _Ctx(lens, starts), q.shape[0]
        ctx.bounds = (256, 4, 2048)
        out = torch.full((n, 8 * dim), 7.0, dtype=torch.bfloat16, device="cuda")
        ops.paged_attention(q.view(n, -1), k, v, tables, ctx, 8, 2, dim, 16, dim ** -0.5, 0, out)
        ops.check_errors()
        want = _want(q, rows, lens, starts, dim ** -0.5, None, 0, None, None, None).view(n, -1)
        assert float((out.double() - want).norm() / want.norm()) < 2.0 ** -8


@pytest.mark.parametrize("dim,packed", [(64, True), (128, True), (64, False), (128, False)])
def test_a_captured_step_without_long_portions_waits_for_the_decode_attention(monkeypatch, dim, packed):
    """Portions of two to four tokens (16 rows and fewer) beside decoded tokens of long contexts: a launch of fixed size holds the prompt
    attention too, none of whose blocks has work.  The product behind it reads what the decode attention writes."""
    from inference_engine_b200.engine.workspace import Workspace
    from inference_engine_b200.kernels import get_ops

    ops, heads, kv_heads = get_ops(), 8, 2
    lens, starts = [2, 1, 4, 3, 1, 1], [5000, 7900, 3001, 6000, 8000, 7000]
    q, k, v, tables, rows = _case(lens, starts, heads, kv_heads, dim, dim, 16, None, 0, dim + 9)
    monkeypatch.setattr(ops, "prompt_packs", lambda *_: packed)
    n, width, out_dim = q.shape[0], heads * dim, 512
    w = torch.randn(out_dim, width, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda").bfloat16()
    attended, ws = torch.zeros(n, width, dtype=torch.bfloat16, device="cuda"), Workspace("cuda", min_rows=n)

    def step(bounds):
        ctx = _Ctx(lens, starts)
        ctx.start_positions, ctx.max_ctx_len, ctx.ws, ctx.bounds = starts, 8001, ws, bounds

        def run():
            ops.paged_attention(q.view(n, -1), k, v, tables, ctx, heads, kv_heads, dim, 16, dim ** -0.5, 0, attended)
            return ops.linear(attended, w, ws=ws, tag="after", out_dtype=torch.float32)

        return ctx, run

    _, eager = step(None)
    eager()
    torch.cuda.synchronize()
    want_rows = attended.double()
    want = want_rows @ w.double().t()
    reference = _want(q, rows, lens, starts, dim ** -0.5, None, 0, None, None, None).view(n, -1)
    assert float((want_rows - reference).norm() / reference.norm()) < 2.0 ** -7
    ctx, run = step((16, 8, 16384))  # (the context stays: its arrays are the captured launches' inputs)
    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run()
    for i in range(50):
        attended.fill_(math.nan)
        graph.replay()
        assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -7, f"replay {i}"
    ops.check_errors()


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("window,keep", [(None, 0), (100, 4)])
@pytest.mark.parametrize("lens,starts,bounds", [([100, 1, 20], [30, 700, 0], (256, 6, 2048)), ([3, 1, 1], [5, 400, 90], (16, 5, 1024)),
                                                ([2, 1], [1000, 0], (32, 4, 1024))])
def test_a_captured_step_with_a_sink(dim, window, keep, lens, starts, bounds):
    """Bounds for more tokens and requests than the step brings: requests beyond its own have no tokens."""
    from inference_engine_b200.kernels import get_ops

    ops, heads, kv_heads, n = get_ops(), 8, 2, sum(lens)
    q, k, v, tables, rows = _case(lens, starts, heads, kv_heads, dim, dim, 16, window, keep, dim)
    extra = bounds[1] - len(lens)
    ctx = _Ctx(lens + [0] * extra, starts + [0] * extra)
    ctx.bounds, ctx.num_tokens = bounds, bounds[0]
    tables = torch.cat([tables, torch.full((extra, tables.shape[1]), -1, dtype=torch.int32, device="cuda")])
    sinks = torch.linspace(-2, 2, heads, device="cuda")
    padded = torch.zeros(bounds[0], heads * dim, dtype=torch.bfloat16, device="cuda")
    padded[:n] = q.view(n, -1)
    out, before = torch.full((bounds[0], heads * dim), 7.0, dtype=torch.bfloat16, device="cuda"), ops.launch_counts.get("sink_attention_packed", 0)
    ops.sink_attention(padded, k, v, tables, ctx, heads, kv_heads, dim, dim, 16, dim ** -0.5, window, sinks, None, out, keep_first=keep)
    ops.check_errors()
    assert ops.launch_counts.get("sink_attention_packed", 0) == before + 1 and bool((out[n:] == 7.0).all())
    want = _want(q, rows, lens, starts, dim ** -0.5, window, keep, None, sinks, None).view(n, -1)
    assert float((out[:n].double() - want).norm() / want.norm()) < REL
