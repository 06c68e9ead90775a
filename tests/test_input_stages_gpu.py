"""Input stages that take rows in pieces of four against the kernels that take them entry by entry: the same sums in another order."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _table(positions, rot_dims):
    angle = torch.arange(positions, device="cuda").float()[:, None] * (10000.0 ** (-torch.arange(0, rot_dims, 2, device="cuda") / rot_dims))
    return torch.stack([angle.cos(), angle.sin()], dim=1).contiguous()


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,rot_dims,interleaved,from_keys", [
    (16, 4, 128, 128, 0, False, False), (5, 1, 64, 64, 64, True, True), (8, 2, 128, 64, 64, False, False), (3, 3, 36, 12, 16, False, False),
    (4, 2, 8, 128, 4, True, False)])
@pytest.mark.parametrize("norm", ["weights", "unit", "values", "none"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_heads_in_pieces_of_four(heads, kv_heads, dim, vdim, rot_dims, interleaved, from_keys, norm, dtype):
    from inference_engine_b200.kernels import get_ops

    ops, n, page = get_ops(), 37, 8
    g = torch.Generator(device="cuda").manual_seed(dim + heads)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    need = (heads + kv_heads) * dim + (0 if from_keys else kv_heads * vdim)
    aligned = rand(n, need + 4)[:, :need] if (need + 4) % 4 == 0 else None
    assert aligned is not None
    ragged = torch.empty(n, need + 5, device="cuda")[:, :need].copy_(aligned)  # rows that no piece of 16 bytes fits: entry by entry
    positions = torch.randint(0, 50, (n,), generator=g, device="cuda", dtype=torch.int32)
    slots = torch.randperm(8 * page, generator=g, device="cuda")[:n].int()
    slots[3] = -1 if norm == "none" else slots[3]  # a slot that is not there
    results = []
    for proj in (aligned, ragged):
        q = torch.zeros(n, heads * dim, dtype=dtype, device="cuda")
        k, v = (torch.zeros(8, kv_heads, page, size, dtype=dtype, device="cuda") for size in (dim, vdim))
        extra = {"bias": (torch.arange(need, device="cuda") % 7 - 3).float() * 0.1, "unit_norm": norm == "unit", "value_norm": norm == "values"}
        if norm == "unit":
            extra.update(q_head_scale=torch.arange(1, heads + 1, device="cuda").float(), warm_coef=0.1, warm_every=8, value_scale=0.5)
        weights = [torch.linspace(0.5, 1.5, dim, device="cuda") for _ in range(2)] if norm == "weights" else [None, None]
        ops.qk_norm_rope_write(proj, positions, _table(50, rot_dims) if rot_dims else None, rot_dims, *weights, 1e-5, q, k, v, slots, heads,
                               kv_heads, dim, vdim, page, values_from_keys=from_keys, interleaved=interleaved, **extra)
        if norm == "none":
            with pytest.raises(Exception, match="page"):
                ops.check_errors()
        else:
            ops.check_errors()
        results.append((q, k, v))
    for a, b in zip(*results):
        # sums of at most 128 squares in another order: 2^-24 sqrt(128) of a value; in bfloat16 some then round the other way, by 2^-8
        torch.testing.assert_close(a.float(), b.float(), rtol=1e-5 if dtype == torch.float32 else 2 ** -7, atol=1e-6)


@pytest.mark.parametrize("heads,dim,rot_dim,rank,rot_dims,interleaved", [(16, 128, 64, 512, 64, True), (3, 64, 32, 256, 16, False), (2, 36, 4, 20, 0, True),
                                                                             (1, 64, 8, 1100, 8, False)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("q_rank", [0, 48, 1536])
def test_latent_rows_of_many_tokens(heads, dim, rot_dim, rank, rot_dims, interleaved, dtype, q_rank):
    """More tokens than four an SM: a warp per token, all that is asked for in one launch.  A few at a time: a block per token.  The bits are the
    same: a token's results do not depend on how many others the step has."""
    from inference_engine_b200.kernels import get_ops

    ops, n, page = get_ops(), 600, 16
    g = torch.Generator(device="cuda").manual_seed(dim)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    q_size, row = heads * (dim + rot_dim), rank + rot_dim
    proj = rand(n, q_size + row + heads + q_rank + (-(heads + row + q_size + q_rank)) % 4)
    positions = torch.randint(0, 700, (n,), generator=g, device="cuda", dtype=torch.int32)
    slots = torch.randperm(40 * page, generator=g, device="cuda")[:n].int()
    table = _table(700, rot_dims) if rot_dims else None
    norm_w, cq_w = rand(rank) * 0.1 + 1, rand(max(q_rank, 1)) * 0.1 + 1
    results = []
    for step in (n, 100):
        plain, absorbed = (torch.zeros(n, heads * size, dtype=dtype, device="cuda") for size in (dim, row))
        gate, cq = torch.zeros(n, heads, device="cuda"), torch.zeros(n, q_rank, dtype=dtype, device="cuda")
        cache = torch.zeros(40, 1, page, row, dtype=dtype, device="cuda")
        for a in range(0, n, step):
            cut = slice(a, a + step)
            part = proj[cut]
            at = q_size + row
            at += (-at) % 4
            extra = dict(cq=part[:, at: at + q_rank], cq_norm_w=cq_w, cq_out=cq[cut]) if q_rank else {}
            ops.latent_prep(positions[cut], table, rot_dims, heads=heads, dim=dim, rot_dim=rot_dim, rank=rank, page_size=page, eps=1e-5,
                            interleaved=interleaved, q=part[:, :q_size], q_plain=plain[cut], q_abs=absorbed[cut],
                            gate_pre=part[:, :heads], gate=gate[cut], dkv=part[:, q_size: q_size + row], norm_w=norm_w, cache=cache,
                            slot_mapping=slots[cut], **extra)
        ops.check_errors()
        results.append((plain, absorbed, gate, cq, cache))
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("lens", [[256], [300, 1, 2, 3, 70], [5] * 60])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,taps", [(4, 4, 128, 128, 4), (4, 2, 64, 256, 3), (8, 8, 36, 20, 2)])
@pytest.mark.parametrize("missing", [False, True])
def test_delta_rule_inputs_of_many_tokens(lens, heads, kv_heads, dim, vdim, taps, missing):
    from types import SimpleNamespace

    from inference_engine_b200.kernels import get_ops
    from inference_engine_b200.kernels.cuda_ops import KernelError

    ops, n, channels = get_ops(), sum(lens), 2 * kv_heads * dim + heads * vdim
    g = torch.Generator(device="cuda").manual_seed(n + dim)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, a, w, rates, bias = rand(n, channels + heads), rand(n, heads * dim), rand(channels, taps), rand(heads), rand(heads * dim)
    state = rand(len(lens), heads * dim * vdim + (taps - 1) * channels)
    ctx = SimpleNamespace(num_seqs=len(lens), cu_q=torch.tensor([0, *lens]).cumsum(0).int().cuda(),
                          seq_of_token=torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).int().cuda())
    slots = torch.randperm(len(lens), generator=torch.Generator().manual_seed(1)).int()
    if missing:
        slots[-1] = len(lens)
    good = n - lens[-1] if missing else n  # (tokens of a request without a slot get anything)
    results = []
    for offset in (0, 1):  # decays that no piece of 16 bytes fits: a thread per channel
        decay = torch.zeros(n * heads * dim + 4, device="cuda")[offset:offset + n * heads * dim].view(n, heads * dim)
        outs = [torch.zeros(n, size, device="cuda") for size in (kv_heads * dim, kv_heads * dim, heads * vdim, heads)] + [decay]
        kept = state.clone()
        ops.delta_prep(x, a, w, rates, bias, kept, slots.cuda(), ctx, *outs, heads, kv_heads, dim, vdim, taps)
        if missing:
            with pytest.raises(KernelError):
                ops.check_errors()
        else:
            ops.check_errors()
        results.append(outs[:4] + [decay.contiguous(), kept])
    for one, other in zip(*results):  # (the same chains of operations)
        assert torch.equal(one[:good], other[:good])


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,taps", [(4, 4, 128, 128, 4), (4, 2, 64, 128, 3), (8, 8, 36, 20, 2)])
def test_delta_rule_inputs_whole_and_in_portions(heads, kv_heads, dim, vdim, taps):
    """700 tokens at once and in portions of 300, 150 and 7: a warp per unit and 8 tokens, tiles of 16, a block per token and unit.  Equal bits."""
    from types import SimpleNamespace

    from inference_engine_b200.kernels import get_ops

    ops, n, channels = get_ops(), 700, 2 * kv_heads * dim + heads * vdim
    g = torch.Generator(device="cuda").manual_seed(dim)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, a, w, rates, bias = rand(n, channels + heads), rand(n, heads * dim), rand(channels, taps), rand(heads), rand(heads * dim)
    state = rand(1, heads * dim * vdim + (taps - 1) * channels)
    results = []
    for step in (700, 300, 150, 7):
        outs, kept = [torch.zeros(n, size, device="cuda") for size in (kv_heads * dim, kv_heads * dim, heads * vdim, heads, heads * dim)], state.clone()
        for at in range(0, n, step):
            cut = slice(at, min(at + step, n))
            ctx = SimpleNamespace(num_seqs=1, cu_q=torch.tensor([0, cut.stop - at], dtype=torch.int32, device="cuda"),
                                  seq_of_token=torch.zeros(cut.stop - at, dtype=torch.int32, device="cuda"))
            ops.delta_prep(x[cut], a[cut], w, rates, bias, kept, torch.zeros(1, dtype=torch.int32, device="cuda"), ctx, *(o[cut] for o in outs),
                           heads, kv_heads, dim, vdim, taps)
        ops.check_errors()
        results.append(outs + [kept])
    for other in results[1:]:
        assert all(torch.equal(one, two) for one, two in zip(results[0], other))


@pytest.mark.parametrize("tokens,channels,rank", [(1, 128, 1), (37, 100, 7), (300, 300, 16), (1000, 2048, 32), (9000, 384, 31), (130, 200, 33)])
@pytest.mark.parametrize("biased", [False, True])
def test_low_rank_decays(tokens, channels, rank, biased):
    """Whatever the tokens a block takes, a number is the same one: as of its token by itself."""
    from inference_engine_b200.kernels import get_ops

    ops, g = get_ops(), torch.Generator(device="cuda").manual_seed(tokens)
    y, w = torch.randn(tokens, rank + 3, generator=g, device="cuda")[:, 2: rank + 2], torch.randn(channels, rank, generator=g, device="cuda")
    bias = torch.randn(channels, generator=g, device="cuda") if biased else None
    out, one = torch.zeros(tokens, channels, device="cuda"), torch.zeros(1, channels, device="cuda")
    ops.lowrank_decay(y, w, bias, 16.0, out)
    x = y.double() @ w.double().T + (0 if bias is None else bias.double())
    # the sum's error (rank + 1 roundings of at most the terms' sizes) through a slope of at most 1 / 16, and a few of the result's own
    size = y.double().abs() @ w.double().abs().T + (0 if bias is None else bias.double().abs())
    assert ((out.double() - torch.exp(torch.nn.functional.logsigmoid(x) / 16)).abs() <= (rank + 1) * 2 ** -24 / 16 * size + 2 ** -21).all()
    for row in {0, tokens // 2, tokens - 1}:
        ops.lowrank_decay(y[row:row + 1], w, bias, 16.0, one)
        assert torch.equal(one[0], out[row])


@pytest.mark.parametrize("heads,vdim", [(16, 128), (7, 36), (5, 4)])
@pytest.mark.parametrize("silu,weighted", [(False, "heads"), (True, "all"), (True, None), (None, "heads")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_rows_in_pieces_of_four(heads, vdim, silu, weighted, dtype):
    from inference_engine_b200.kernels import get_ops

    ops, tokens = get_ops(), 2501
    g = torch.Generator(device="cuda").manual_seed(vdim)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    rows, wide = rand(tokens * heads * vdim), rand(tokens, heads * vdim + 8)
    weight = None if weighted is None else rand(heads * vdim if weighted == "heads" else vdim)
    results = []
    for offset in (0, 1):  # rows that no piece of 16 bytes fits: an entry a lane at a time
        o = torch.empty(rows.numel() + 4, device="cuda")[offset:offset + rows.numel()].copy_(rows).view(tokens, heads * vdim)
        out = torch.zeros(tokens, heads * vdim, dtype=dtype, device="cuda")
        gate = None if silu is None else wide[:, 4: 4 + heads * vdim]
        ops.recurrence_readout(o, None, weight, 1e-5, gate, out, heads, vdim, vdim, gate_act="silu" if silu else "sigmoid")
        results.append(out.float())
    assert torch.equal(*results)  # (the same chains of operations)
    # and so a row's result does not depend on how many there are
    few = torch.zeros(3, heads * vdim, dtype=dtype, device="cuda")
    ops.recurrence_readout(rows.view(tokens, -1)[1700:1703], None, weight, 1e-5, None if gate is None else gate[1700:1703], few, heads, vdim, vdim,
                           gate_act="silu" if silu else "sigmoid")
    assert torch.equal(few.float(), results[0][1700:1703])


@pytest.mark.parametrize("heads,vdim", [(16, 128), (7, 36), (3, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_heads_of_many_and_of_few_tokens(heads, vdim, dtype):
    """The delta rule's read-out: the same bits for a token among 2,501 and among 3."""
    from inference_engine_b200.kernels import get_ops

    ops, tokens = get_ops(), 2501
    g = torch.Generator(device="cuda").manual_seed(vdim)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    o, gate, weight = rand(tokens, heads * vdim), rand(tokens, heads * vdim), rand(vdim)
    out, few = torch.zeros(tokens, heads * vdim, dtype=dtype, device="cuda"), torch.zeros(3, heads * vdim, dtype=dtype, device="cuda")
    ops.gated_rms_heads(o, weight, 1e-5, gate, out, heads, vdim)
    ops.gated_rms_heads(o[900:903], weight, 1e-5, gate[900:903], few, heads, vdim)
    assert torch.equal(out[900:903], few)
