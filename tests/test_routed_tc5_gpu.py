"""The routed feed-forward's grouped products on tcgen05 against plain sums in 64 bits, over tile edges and ragged widths."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(x, ids, weights, gate_up, down, limit, alpha, offset):
    from inference_engine_b200.engine.workspace import Workspace
    from inference_engine_b200.kernels import get_ops

    ops = get_ops()
    before = ops.launch_counts.get("routed_tc5_down", 0)
    out = ops.routed_experts(x, ids, weights, gate_up, down, limit=limit, alpha=alpha, up_offset=offset, ws=Workspace("cuda"))
    ops.check_errors()
    return out, ops.launch_counts.get("routed_tc5_down", 0) - before


def _want(x, ids, weights, gate_up, down, limit, alpha, offset):
    n, top = ids.shape
    out = torch.zeros(top, n, x.shape[1], dtype=torch.float64, device=x.device)
    for e in range(gate_up.shape[0]):
        token, choice = (ids == e).nonzero(as_tuple=True)
        rows = x[token].double()
        g, u = rows @ gate_up[e, 0].double().T, rows @ gate_up[e, 1].double().T
        if limit is not None:
            g, u = g.clamp(max=limit), u.clamp(-limit, limit)
        y = (g * torch.sigmoid(alpha * g) * (u + offset)).bfloat16().double()
        out[choice, token] = (y @ down[e].double().T) * weights[token, choice].double()[:, None]
    return out


# pairs per expert: around the rounding to 16, the largest tile, and several tiles; experts nobody chose
@pytest.mark.parametrize("counts", [[0, 1, 15, 16, 17, 63], [255, 256, 257, 0, 513, 64], [0, 0, 1400, 0, 0, 0], [3] * 5 + [9]])
@pytest.mark.parametrize("hidden,ff,limit", [(128, 64, None), (320, 136, 1.5), (72, 264, None), (512, 128, 0.7)])
def test_pairs_per_expert(counts, hidden, ff, limit):
    g = torch.Generator(device="cuda").manual_seed(hidden + len(counts))
    experts, n, top = len(counts), sum(counts), 1
    ids = torch.repeat_interleave(torch.arange(experts), torch.tensor(counts))[torch.randperm(n)].view(n, top).int().cuda()
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, gate_up, down = rand(n, hidden).bfloat16(), (rand(experts, 2, ff, hidden) * hidden ** -0.5).bfloat16(), (rand(experts, hidden, ff) * ff ** -0.5).bfloat16()
    args = (x, ids, torch.rand(n, top, generator=g, device="cuda"), gate_up, down, limit, 1.3, 0.5)
    got, ran = _run(*args)
    assert ran == 1
    # y is rounded to 8 bits in both, from sums that differ in the last of 24: a few roundings fall the other way
    want = _want(*args)
    torch.testing.assert_close(got.double(), want, atol=2e-2, rtol=1e-2)
    assert float((got.double() - want).norm() / want.norm()) < 1e-3


@pytest.mark.parametrize("tokens,top,experts", [(2600, 4, 8), (33, 2, 4), (301, 3, 40)])
def test_several_choices_per_token(tokens, top, experts):
    """More pairs than the sorting block keeps in registers (8,192); the order among an expert's pairs changes nothing."""
    g = torch.Generator(device="cuda").manual_seed(tokens)
    hidden, ff = 64, 64
    ids = torch.rand(tokens, experts, generator=g, device="cuda").topk(top, dim=-1).indices.int()
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, gate_up, down = rand(tokens, hidden).bfloat16(), (rand(experts, 2, ff, hidden) * 0.1).bfloat16(), (rand(experts, hidden, ff) * 0.1).bfloat16()
    args = (x, ids, torch.rand(tokens, top, generator=g, device="cuda"), gate_up, down, None, 1.0, 0.0)
    got, ran = _run(*args)
    assert ran == 1
    want = _want(*args)
    assert float((got.double() - want).norm() / want.norm()) < 1e-3
    assert torch.equal(got, _run(*args)[0])
