"""The recurrences in chunks of 64 tokens against the plain ones in 64 bits, and against the kernels that go token by token."""

import pytest
import torch

from tests.ref_ops import RefOps

pytestmark = pytest.mark.gpu

# 32-bit sums of at most 128 + 64 terms and products of at most 64 decays: 2^-24 (sqrt(192) + sqrt(64)) is 1.3e-6 of a sum's
# terms; outputs in which terms cancel lose a little more.
REL = 4e-6


class _Ctx:
    def __init__(self, lens, device):
        from inference_engine_b200.engine.workspace import Workspace

        starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
        self.q_starts, self.q_lens, self.num_seqs, self.max_q_len = starts[:-1], lens, len(lens), max(lens)
        self.cu_q = torch.tensor(starts, dtype=torch.int32, device=device)
        self.ws = Workspace(device)


@pytest.fixture
def ops(monkeypatch):
    from inference_engine_b200.kernels import get_ops

    monkeypatch.setattr(get_ops(), "chunks_always", True)
    return get_ops()


def _close(got, want, what):
    rel = float((got.double().cpu() - want.double()).norm() / want.double().norm())
    assert rel < REL, f"{what}: {rel:.2e}"


LENS = [[64], [65, 1, 63], [7, 200, 0, 129], [300]]
SIZES = [(2, 128, 128), (40, 128, 128), (3, 64, 64), (1, 128, 64), (2, 64, 100), (2, 40, 12), (1, 96, 260)]


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("heads,dim,vdim", SIZES)
def test_decays_per_channel(ops, heads, dim, vdim, lens):
    g, n = torch.Generator().manual_seed(dim + vdim), sum(lens)
    pad = torch.randn(n, 2 * heads * dim + heads * vdim + 4, generator=g)  # (views of one projection)
    decay = torch.sigmoid(torch.randn(n, heads * dim, generator=g) * 2 + 3)
    decay[::37, ::5] = 0.0  # whatever was there is forgotten
    state = torch.randn(6, heads * vdim * dim + 3, generator=g)
    slots = torch.tensor([3, 0, 5, 1][: len(lens)], dtype=torch.int32)
    qk = heads * dim
    want_state, want = state.double(), torch.zeros(n, heads * vdim, dtype=torch.float64)
    cut = lambda t: (t[:, :qk], t[:, qk: 2 * qk], t[:, 2 * qk: 2 * qk + heads * vdim])  # noqa: E731
    q, w, v = cut(pad.double())
    RefOps().gated_recurrence(q, decay.double(), w, None, v, want_state, slots, _Ctx(lens, "cpu"), want, heads, dim, vdim, vdim, 0.3)
    got_state, got, ctx = state.cuda(), torch.zeros(n, heads * vdim, device="cuda"), _Ctx(lens, "cuda")
    q, w, v = cut(pad.cuda())
    before = ops.launch_counts.get("gated_recurrence_chunks", 0)
    ops.gated_recurrence(q, decay.cuda(), w, None, v, got_state, slots.cuda(), ctx, got, heads, dim, vdim, vdim, 0.3, in_chunks=True)
    assert ops.launch_counts.get("gated_recurrence_chunks", 0) == before + 1
    _close(got, want, "outputs")
    _close(got_state, want_state, "states")
    for s in set(range(6)) - set(slots.tolist()):
        assert torch.equal(got_state[s].cpu(), state[s])


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("heads,dim,vdim,normaliser,unit", [(2, 128, 128, 1, 1), (4, 64, 64, 1, 1), (2, 48, 20, 1, 1), (4, 128, 64, 0, 2)])
def test_decays_per_head(ops, heads, dim, vdim, normaliser, unit, lens):
    g, n, cols = torch.Generator().manual_seed(dim + vdim), sum(lens), vdim + normaliser
    q, w = (torch.randn(n, heads // unit * dim, generator=g) for _ in range(2))
    v = torch.randn(n, heads * vdim, generator=g)
    gates = torch.rand(n, heads, 3, generator=g) * 0.4 + 0.6
    gates[:: 50, 0, 0] = 0.0
    state, slots = torch.randn(6, heads * cols * dim, generator=g), torch.tensor([3, 0, 5, 1][: len(lens)], dtype=torch.int32)
    want_state, want = state.double(), torch.zeros(n, heads * cols, dtype=torch.float64)
    RefOps().gated_recurrence(q.double(), None, w.double(), gates.double(), v.double(), want_state, slots, _Ctx(lens, "cpu"), want,
                              heads, dim, vdim, cols, 0.1, heads_per_unit=unit)
    got_state, got = state.cuda(), torch.zeros(n, heads * cols, device="cuda")
    ops.gated_recurrence(q.cuda(), None, w.cuda(), gates.cuda(), v.cuda(), got_state, slots.cuda(), _Ctx(lens, "cuda"), got, heads,
                         dim, vdim, cols, 0.1, heads_per_unit=unit, in_chunks=True)
    _close(got, want, "outputs")
    _close(got_state, want_state, "states")


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(2, 2, 128, 128), (4, 2, 64, 64), (2, 1, 128, 36), (2, 2, 24, 128)])
def test_delta_rule(ops, heads, kv_heads, dim, vdim, lens):
    g, n = torch.Generator().manual_seed(dim + vdim), sum(lens)
    unit = lambda t: t / t.norm(dim=-1, keepdim=True)  # noqa: E731
    q = (unit(torch.randn(n, kv_heads, dim, generator=g)) * dim ** -0.5).view(n, -1)
    k = unit(torch.randn(n, kv_heads, dim, generator=g) + 0.5).view(n, -1)  # (keys that resemble each other)
    v, beta = torch.randn(n, heads * vdim, generator=g), torch.sigmoid(torch.randn(n, heads, generator=g) + 1)
    decay = torch.sigmoid(torch.randn(n, heads * dim, generator=g) + 4)
    decay[::41, ::3] = 0.0
    state, slots = torch.randn(6, heads * vdim * dim + 5, generator=g), torch.tensor([3, 0, 5, 1][: len(lens)], dtype=torch.int32)
    want_state, want = state.double(), torch.zeros(n, heads * vdim, dtype=torch.float64)
    args = (q, k, v, beta, decay)
    RefOps().delta_rule(*(t.double() for t in args), want_state, slots, _Ctx(lens, "cpu"), want, heads, kv_heads, dim, vdim)
    got_state, got = state.cuda(), torch.zeros(n, heads * vdim, device="cuda")
    before = ops.launch_counts.get("delta_rule_chunks", 0)
    ops.delta_rule(*(t.cuda() for t in args), got_state, slots.cuda(), _Ctx(lens, "cuda"), got, heads, kv_heads, dim, vdim, in_chunks=True)
    assert ops.launch_counts.get("delta_rule_chunks", 0) == before + 1
    _close(got, want, "outputs")
    _close(got_state, want_state, "states")


@pytest.mark.parametrize("dim,vdim", [(30, 32), (130, 64), (64, 33)])
def test_other_sizes_go_token_by_token(ops, dim, vdim):
    """Sizes without whole 16-byte pieces, and key sizes above 128."""
    n, heads, lens = 70, 2, [70]
    q, w, decay = (torch.rand(n, heads * dim, device="cuda") for _ in range(3))
    v, state = torch.rand(n, heads * vdim, device="cuda"), torch.zeros(2, heads * vdim * dim, device="cuda")
    outs = []
    for in_chunks in (False, True):
        out, st = torch.zeros(n, heads * vdim, device="cuda"), state.clone()
        ops.gated_recurrence(q, decay, w, None, v, st, torch.tensor([1], dtype=torch.int32, device="cuda"), _Ctx(lens, "cuda"), out,
                             heads, dim, vdim, vdim, 1.0, in_chunks=in_chunks)
        outs.append((out, st))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


def test_a_value_that_is_no_number_reaches_no_earlier_token(ops):
    n, heads, dim, vdim = 150, 1, 128, 128
    g = torch.Generator().manual_seed(3)
    q, w = (torch.randn(n, heads * dim, generator=g).cuda() for _ in range(2))
    v, decay = torch.randn(n, heads * vdim, generator=g).cuda(), torch.rand(n, heads * dim, generator=g).cuda()
    v[77] = float("nan")
    out, state = torch.zeros(n, heads * vdim, device="cuda"), torch.zeros(1, heads * vdim * dim, device="cuda")
    ops.gated_recurrence(q, decay, w, None, v, state, torch.zeros(1, dtype=torch.int32, device="cuda"), _Ctx([n], "cuda"), out, heads,
                         dim, vdim, vdim, 1.0, in_chunks=True)
    assert torch.isfinite(out[:77]).all() and torch.isnan(out[77:]).all()


@pytest.mark.parametrize("rule", ["decays", "delta"])
@pytest.mark.parametrize("lens", [[7, 200, 129], [65], [1, 1, 64, 300]])
@pytest.mark.parametrize("bounds,most", [((512, 6, 1024), 512), ((1024, 16, 4096), 512)])
def test_a_launch_for_bounds_serves_every_step_within_them(ops, rule, lens, bounds, most):
    """A captured step: tokens beyond the step's own belong to no request, requests beyond them have none; blocks for chunks that
    the step does not have leave.  The bits are those of a launch for the step itself."""
    heads, dim, vdim, n = 3, 64, 128, sum(lens)
    g = torch.Generator().manual_seed(n)
    tokens, seqs, _ = bounds
    rand = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    pad = lambda t: torch.cat([t, rand(tokens - n, t.shape[1])]).cuda()  # noqa: E731
    q, k, v, decay = rand(n, heads * dim) * 0.2, rand(n, heads * dim) * 0.2, rand(n, heads * vdim), torch.rand(n, heads * dim, generator=g)
    beta = torch.rand(n, heads, generator=g)
    state = rand(seqs + 1, heads * vdim * dim)
    results = []
    for captured in (False, True):
        args = [pad(t) if captured else t.cuda() for t in (q, k, v, decay, beta)]
        ctx = _Ctx(lens + [0] * (seqs - len(lens) if captured else 0), "cuda")
        if captured:
            ctx.bounds, ctx.most_portion = bounds, most
        slots = torch.tensor(list(range(len(lens))) + [seqs] * (ctx.num_seqs - len(lens)), dtype=torch.int32, device="cuda")
        st, out = state.cuda(), torch.full((args[0].shape[0], heads * vdim), 7.0, device="cuda")
        counts = dict(ops.launch_counts)
        if rule == "delta":
            ops.delta_rule(args[0], args[1], args[2], args[4], args[3], st, slots, ctx, out, heads, heads, dim, vdim, in_chunks=True)
        else:
            ops.gated_recurrence(args[0], args[3], args[1], None, args[2], st, slots, ctx, out, heads, dim, vdim, vdim, 0.5, in_chunks=True)
        name = "delta_rule_chunks" if rule == "delta" else "gated_recurrence_chunks"
        assert ops.launch_counts.get(name, 0) == counts.get(name, 0) + 1
        assert (out[n:] == 7.0).all()
        results.append((out[:n], st))
    ops.check_errors()
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("what", ["v", "k"])
@pytest.mark.parametrize("dim,vdim", [(128, 128), (64, 36)])
def test_delta_rule_with_a_value_that_is_no_number(ops, value, what, dim, vdim):
    """It reaches no earlier token, also of its own sixteen, and those come out as without it."""
    n, heads, at = 150, 2, 77
    g = torch.Generator().manual_seed(3)
    rand = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    unit = lambda t: t / t.norm(dim=-1, keepdim=True)  # noqa: E731
    q, k = (unit(rand(n, heads, dim)).view(n, -1) for _ in range(2))
    v, beta, decay = rand(n, heads * vdim), torch.sigmoid(rand(n, heads)), torch.sigmoid(rand(n, heads * dim) + 4)
    outs = []
    for spoilt in (False, True):
        if spoilt:
            (v if what == "v" else k)[at, :3] = value
        out, state = torch.zeros(n, heads * vdim, device="cuda"), torch.zeros(1, heads * vdim * dim, device="cuda")
        ops.delta_rule(q, k, v, beta, decay, state, torch.zeros(1, dtype=torch.int32, device="cuda"), _Ctx([n], "cuda"), out, heads, heads, dim,
                       vdim, in_chunks=True)
        outs.append(out)
    assert torch.isfinite(outs[0]).all() and torch.isfinite(outs[1][:at]).all()
    assert not torch.isfinite(outs[1][at:, :3]).all(dim=1).any()
    # (the spoilt chunk goes token by token: the same sums in another order)
    assert float((outs[0][:at] - outs[1][:at]).norm() / outs[0][:at].norm()) < REL


@pytest.mark.parametrize("where", ["value", "key", "query", "state"])
@pytest.mark.parametrize("dim,vdim,gated", [(128, 128, False), (64, 36, False), (64, 64, True)])
def test_infinities_stay_infinities(ops, where, dim, vdim, gated):
    """Positive numbers, one of them infinite: what is infinite token by token is so in chunks, for all later tokens, and nothing else changes."""
    n, heads, at, cols = 150, 2, 70, vdim + gated
    g = torch.Generator().manual_seed(5)
    rand = lambda *s: (torch.rand(*s, generator=g) + 0.1).cuda()  # noqa: E731
    q, w, v, decay, gates = rand(n, heads * dim), rand(n, heads * dim), rand(n, heads * vdim), rand(n, heads * dim) * 0.5 + 0.4, rand(n, heads, 3) * 0.5 + 0.4
    state = rand(1, heads * cols * dim)
    ({"value": v, "key": w, "query": q, "state": state}[where])[0 if where == "state" else at, 7] = float("inf")
    results = []
    for in_chunks in (False, True):
        out, st = torch.zeros(n, heads * cols, device="cuda"), state.clone()
        ops.gated_recurrence(q, None if gated else decay, w, gates if gated else None, v, st, torch.zeros(1, dtype=torch.int32, device="cuda"),
                             _Ctx([n], "cuda"), out, heads, dim, vdim, cols, 0.5, in_chunks=in_chunks)
        results.append(out)
    one, chunks = results
    assert not torch.isnan(one).any() and torch.isinf(one).any()
    assert torch.equal(torch.isinf(one), torch.isinf(chunks)) and not torch.isnan(chunks).any()
    good = torch.isfinite(one)
    assert float((one[good] - chunks[good]).norm() / one[good].norm()) < REL
