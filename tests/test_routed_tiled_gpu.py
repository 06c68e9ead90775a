"""The routed feed-forward on weights laid out in tiles against plain sums in 64 bits: edges of the tiles of pairs, ragged widths, few
tokens and many; and the router's products on the tensor cores."""

import pytest
import torch

from tests.test_routed_tc5_gpu import _want

pytestmark = pytest.mark.gpu


def _run(x, ids, weights, gate_up, down, limit, alpha, offset):
    from inference_engine_b200.engine.workspace import Workspace
    from inference_engine_b200.kernels import get_ops
    from inference_engine_b200.parts.routed import ExpertTiles

    ops = get_ops()
    before = dict(ops.launch_counts)
    out = ops.routed_experts_tiled(x, ids, weights, ExpertTiles.of(gate_up, down), limit=limit, alpha=alpha, up_offset=offset, ws=Workspace("cuda"))
    ops.check_errors()
    return out, {name for name, n in ops.launch_counts.items() if n > before.get(name, 0)}


# pairs per expert: around the rounding to 32, an accumulator's 256, a tile's 320, several tiles; experts nobody chose; up to 64 tokens
@pytest.mark.parametrize("counts", [[0, 1, 31, 32, 33, 63], [255, 256, 257, 0, 320, 64], [319, 321, 640, 641, 0, 8], [383, 384, 385, 0, 770, 8], [0, 0, 2300, 0], [1, 0, 15, 16, 17],
                                    [0, 64, 0], [1]])
@pytest.mark.parametrize("hidden,ff,limit", [(128, 64, None), (320, 136, 1.5), (72, 264, None), (520, 128, 0.7)])
def test_pairs_per_expert(counts, hidden, ff, limit):
    g = torch.Generator(device="cuda").manual_seed(hidden + len(counts))
    experts, n, top = len(counts), sum(counts), 1
    ids = torch.repeat_interleave(torch.arange(experts), torch.tensor(counts))[torch.randperm(n)].view(n, top).int().cuda()
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, gate_up, down = rand(n, hidden).bfloat16(), (rand(experts, 2, ff, hidden) * hidden ** -0.5).bfloat16(), (rand(experts, hidden, ff) * ff ** -0.5).bfloat16()
    args = (x, ids, torch.rand(n, top, generator=g, device="cuda"), gate_up, down, limit, 1.3, 0.5)
    got, ran = _run(*args)
    assert ("routed_few_down" if n <= 64 else "routed_pair_down") in ran
    # y is rounded to 8 bits in both, from sums that differ in the last of 24: a few roundings fall the other way
    want = _want(*args)
    torch.testing.assert_close(got.double(), want, atol=2e-2, rtol=1e-2)
    assert float((got.double() - want).norm() / want.norm()) < 1e-3


@pytest.mark.parametrize("tokens,top,experts", [(2600, 4, 8), (33, 2, 4), (64, 3, 40), (65, 3, 40), (301, 3, 40)])
@pytest.mark.parametrize("aligned", [True, False])
def test_several_choices_per_token(tokens, top, experts, aligned):
    """More pairs than the sorting block keeps in registers (8,192); rows that start anywhere; an id that is no expert."""
    g = torch.Generator(device="cuda").manual_seed(tokens)
    hidden, ff = 64, 72
    ids = torch.rand(tokens, experts, generator=g, device="cuda").topk(top, dim=-1).indices.int()
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x = rand(tokens * hidden + 8).bfloat16()[0 if aligned else 1:][: tokens * hidden].view(tokens, hidden)
    gate_up, down = (rand(experts, 2, ff, hidden) * 0.1).bfloat16(), (rand(experts, hidden, ff) * 0.1).bfloat16()
    args = (x, ids, torch.rand(tokens, top, generator=g, device="cuda"), gate_up, down, None, 1.0, 0.0)
    got, want = _run(*args)[0], _want(*args)
    assert float((got.double() - want).norm() / want.norm()) < 1e-3
    ids[5, 0] = experts
    got, want = _run(*args)[0], _want(*args)
    got[0, 5] = want[0, 5] = 0.0  # (a pair without an expert is nobody's)
    assert float((got.double() - want).norm() / want.norm()) < 1e-3


@pytest.mark.parametrize("tokens,width,experts,top,groups,keep", [(600, 64, 7, 2, 1, 1), (1000, 2048, 32, 4, 4, 2), (593, 288, 40, 3, 8, 3), (2048, 96, 64, 4, 1, 1)])
@pytest.mark.parametrize("scoring", ["softmax", "sigmoid"])
def test_router_of_many_tokens(tokens, width, experts, top, groups, keep, scoring):
    from inference_engine_b200.kernels import get_ops

    ops, g = get_ops(), torch.Generator(device="cuda").manual_seed(width)
    x = torch.randn(tokens, width, generator=g, device="cuda").bfloat16()
    w = torch.randn(experts, width, generator=g, device="cuda") * width ** -0.5
    bias = torch.randn(experts, generator=g, device="cuda") * 0.1
    correction = torch.randn(experts, generator=g, device="cuda") * 0.01 if scoring == "sigmoid" else None
    ids, weights = torch.empty(tokens, top, dtype=torch.int32, device="cuda"), torch.empty(tokens, top, device="cuda")
    ops.route_topk(x, w, groups, keep, ids, weights, bias=bias, scoring=scoring, correction=correction)
    logits = x.double() @ w.double().T + bias.double()
    scores = logits.softmax(-1) if scoring == "softmax" else logits.sigmoid()
    choice = scores + (correction.double() if correction is not None else 0)
    best = choice.view(tokens, groups, -1).amax(-1)
    kept = torch.zeros(tokens, groups, dtype=torch.bool, device="cuda").scatter_(1, best.topk(keep, dim=-1).indices, True)
    allowed = choice.masked_fill(~kept.repeat_interleave(experts // groups, dim=1), -1.0)
    ranked = allowed.sort(dim=-1, descending=True)
    # sums of 32 bits: where two scores (or two groups) are further apart than 1e-5 the choice is the same
    gap = (ranked.values[:, :top] - ranked.values[:, 1: top + 1]).amin(-1) if top < experts else torch.ones(tokens, device="cuda")
    if keep < groups:
        by_group = best.sort(dim=-1, descending=True).values
        gap = torch.minimum(gap, by_group[:, keep - 1] - by_group[:, keep])
    sure = gap > 1e-5
    assert sure.float().mean() > 0.97
    assert torch.equal(ids[sure].long(), ranked.indices[sure, :top])
    want = scores.gather(1, ids.long())
    want = want / want.sum(-1, keepdim=True)
    torch.testing.assert_close(weights[sure].double(), want[sure], atol=2e-6, rtol=2e-5)


# around the room for 64 pairs of the kernel for few tokens, and for as many pairs as a step has tokens of the other one
@pytest.mark.parametrize("tokens", [1, 8, 16, 17, 20, 33, 62, 64, 65, 100, 256, 257, 300])
@pytest.mark.parametrize("repeats", ["one expert", "twice each"])
def test_tokens_that_name_an_expert_more_than_once(tokens, repeats):
    g = torch.Generator(device="cuda").manual_seed(tokens)
    experts, top, hidden, ff = 5, 4, 136, 72
    if repeats == "one expert":
        ids = torch.zeros(tokens, top, dtype=torch.int32, device="cuda")
    else:
        ids = torch.randint(0, experts, (tokens, 2), generator=g, device="cuda", dtype=torch.int32).repeat(1, 2)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, gate_up, down = rand(tokens, hidden).bfloat16(), (rand(experts, 2, ff, hidden) * 0.1).bfloat16(), (rand(experts, hidden, ff) * 0.1).bfloat16()
    args = (x, ids, torch.rand(tokens, top, generator=g, device="cuda"), gate_up, down, None, 1.0, 0.0)
    got, ran = _run(*args)
    assert ("routed_few_down" if tokens <= 64 else "routed_pair_down") in ran
    want = _want(*args)
    assert float((got.double() - want).norm() / want.norm()) < 1e-3


@pytest.mark.parametrize("tokens", [8, 20, 62, 64, 65, 100, 256, 300, 700])
@pytest.mark.parametrize("spoilt", ["one", "most", "all"])
@pytest.mark.parametrize("scoring", ["softmax", "sigmoid"])
def test_rows_that_are_no_numbers(tokens, spoilt, scoring):
    """Routing gives them expert 0 for every choice.  The other rows come out as beside good ones, bit for bit."""
    from inference_engine_b200.kernels import get_ops

    ops, g = get_ops(), torch.Generator(device="cuda").manual_seed(tokens)
    experts, top, hidden, ff = 6, 4, 192, 64
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, router = rand(tokens, hidden).bfloat16(), rand(experts, hidden) * hidden ** -0.5
    gate_up, down = (rand(experts, 2, ff, hidden) * 0.1).bfloat16(), (rand(experts, hidden, ff) * 0.1).bfloat16()
    bad = torch.zeros(tokens, dtype=torch.bool, device="cuda")
    bad[{"one": slice(tokens // 2, tokens // 2 + 1), "most": slice(3, None), "all": slice(None)}[spoilt]] = True
    outs = []
    for rows in (x, x.masked_fill(bad[:, None], float("nan"))):
        ids, weights = torch.empty(tokens, top, dtype=torch.int32, device="cuda"), torch.empty(tokens, top, device="cuda")
        ops.route_topk(rows, router, 1, 1, ids, weights, scoring=scoring)
        outs.append(_run(rows, ids, weights, gate_up, down, None, 1.0, 0.0)[0])
    assert (ids[bad] == 0).all()
    assert torch.isfinite(outs[0]).all() and torch.equal(outs[0][:, ~bad], outs[1][:, ~bad])
    assert not torch.isfinite(outs[1][:, bad]).any()


@pytest.mark.parametrize("scoring", ["softmax", "sigmoid"])
def test_router_of_many_tokens_with_infinities(scoring):
    """An infinite activation gives infinite logits, and a choice, as among few tokens; a weight that rounds beyond bfloat16's range is one like others."""
    from inference_engine_b200.kernels import get_ops

    ops, g = get_ops(), torch.Generator(device="cuda").manual_seed(2)
    tokens, width, experts, top = 700, 256, 12, 3
    x = torch.randn(tokens, width, generator=g, device="cuda").bfloat16()
    w = torch.randn(experts, width, generator=g, device="cuda") * width ** -0.5
    w[:, 9] = torch.arange(experts, device="cuda") % 2 * 2.0 - 1  # no lower parts
    w[2, 5], w[7, 6] = 3.4028234e38, float("-inf")
    x[:, 5], x[300:, 6] = 0.0, 0.0
    x[:300, 6] = x[:300, 6].abs() + 1
    x[3, 7], x[17, 100], x[18, 9], x[650, 9] = float("inf"), float("-inf"), float("inf"), float("nan")
    x[40, 8], x[40, 9] = float("inf"), float("-inf")
    correction = torch.randn(experts, generator=g, device="cuda") * 0.01 if scoring == "sigmoid" else None
    results = []
    for step in (700, 100):
        ids, weights = torch.full((tokens, top), -1, dtype=torch.int32, device="cuda"), torch.empty(tokens, top, device="cuda")
        for at in range(0, tokens, step):
            ops.route_topk(x[at: at + step], w, 1, 1, ids[at: at + step], weights[at: at + step], scoring=scoring, correction=correction)
        results.append((ids, weights))
    (many, many_weights), (few, few_weights) = results
    assert torch.equal(many, few)
    # logits of 32-bit sums in another order
    torch.testing.assert_close(many_weights, few_weights, atol=2e-6, rtol=2e-5, equal_nan=True)
    if scoring == "sigmoid":
        assert len(set(few[17].tolist())) == top and len(set(few[18].tolist())) == top  # (a choice, not expert 0 for all)


@pytest.mark.parametrize("tokens,experts", [(64, 1), (2048, 8)])
def test_the_activation_is_a_32_bit_one(tokens, experts):
    """Rows with a single 1 and identities as down matrices, so that gates, ups and what becomes of them are seen as they are.  An exponential of at most
    two units in the last place and three more roundings leave 2^-22 + 3 * 2^-24 of a value; where that crosses no boundary between two
    bfloat16 numbers the result is the one that 64 bits round to."""
    g, size = torch.Generator(device="cuda").manual_seed(tokens), 256
    gate = (torch.rand(experts, size, size, generator=g, device="cuda") * 80 - 60).bfloat16()
    up = torch.randn(experts, size, size, generator=g, device="cuda").bfloat16()
    down = torch.eye(size, device="cuda").bfloat16().repeat(experts, 1, 1)
    at = torch.arange(tokens, device="cuda")
    x = torch.zeros(tokens, size, device="cuda", dtype=torch.bfloat16)
    x[at, at % size] = 1.0
    ids = (at // size).int()[:, None]
    got = _run(x, ids, torch.ones(tokens, 1, device="cuda"), torch.stack([gate, up], dim=1), down, None, 1.0, 0.0)[0][0]
    a, u = (m.transpose(1, 2).reshape(-1, size)[:tokens].double() for m in (gate, up))
    want = a / (1 + torch.exp(-a)) * u
    room = 7 * 2.0 ** -24
    low, high = (want * (1 - room)).bfloat16(), (want * (1 + room)).bfloat16()
    assert ((got == low.float()) | (got == high.float())).all()


@pytest.mark.parametrize("width,experts", [(2048, 32), (1024, 16)])
@pytest.mark.parametrize("weights_of", [torch.float32, torch.bfloat16])
def test_router_of_many_tokens_is_as_exact_as_that_of_few(width, experts, weights_of):
    """Both kernels' weights against 64 bits, over eight draws; a hundredth more for the draws' own spread."""
    from inference_engine_b200.kernels import get_ops

    ops, tokens, errors = get_ops(), 1000, [0.0, 0.0]
    for seed in range(8):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn(tokens, width, generator=g, device="cuda").bfloat16()
        w = (torch.randn(experts, width, generator=g, device="cuda") * 0.02).to(weights_of).float()
        scores = (x.double() @ w.double().T).softmax(-1)
        for i, step in enumerate((tokens, 500)):
            ids, weights = torch.empty(tokens, experts, dtype=torch.int32, device="cuda"), torch.empty(tokens, experts, device="cuda")
            for at in range(0, tokens, step):
                ops.route_topk(x[at: at + step], w, 1, 1, ids[at: at + step], weights[at: at + step])
            want = scores.gather(1, ids.long())
            errors[i] += float((weights.double() - want).norm() / want.norm())
    assert errors[0] < 1.01 * errors[1]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width,experts", [(192, 5), (1028, 40), (50, 3)])
def test_router_of_one_to_four_tokens_an_sm(dtype, width, experts):
    """Blocks of 1,024 threads, one an SM, and (bfloat16) of 256, up to four: the same bits for a token among any number."""
    from inference_engine_b200.kernels import get_ops

    ops, g = get_ops(), torch.Generator(device="cuda").manual_seed(width)
    top, sms = 2, torch.cuda.get_device_properties(0).multi_processor_count
    x = torch.randn(4 * sms - 1, width, generator=g, device="cuda").to(dtype)
    w = torch.randn(experts, width, generator=g, device="cuda") * width ** -0.5

    def route(rows):
        ids, weights = torch.empty(rows.shape[0], top, dtype=torch.int32, device="cuda"), torch.empty(rows.shape[0], top, device="cuda")
        ops.route_topk(rows, w, 1, 1, ids, weights, scoring="sigmoid")
        return ids, weights

    ids, weights = route(x)
    ranked = (x.double() @ w.double().T).sigmoid().sort(dim=-1, descending=True)
    sure = (ranked.values[:, 0] - ranked.values[:, 1] > 1e-5) & (ranked.values[:, 1] - ranked.values[:, 2] > 1e-5)
    assert sure.float().mean() > 0.97 and torch.equal(ids[sure].long(), ranked.indices[sure, :top])
    for tokens in (1, sms, sms + 1, 2 * sms, 2 * sms + 1, 3 * sms, 3 * sms + 1):
        some = route(x[:tokens])
        assert torch.equal(some[0], ids[:tokens]) and torch.equal(some[1], weights[:tokens])
