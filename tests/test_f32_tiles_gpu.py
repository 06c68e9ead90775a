"""The 32-bit path's tiled kernels give the bits that its row-by-row kernels give, whatever the tiles."""

import pytest
import torch

from tests.test_attention_packed_gpu import _Ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [32, 64, 128])
@pytest.mark.parametrize("heads,kv_heads", [(4, 4), (6, 2), (8, 1)])
@pytest.mark.parametrize("lens,starts", [([16], [0]), ([33, 1, 70], [0, 77, 31]), ([100], [200])])
@pytest.mark.parametrize("window,page", [(0, 16), (1, 8), (40, 16), (33, 1)])
def test_attention_is_bit_for_bit_the_general_one(hd, heads, kv_heads, lens, starts, window, page):
    from inference_engine_b200.kernels import get_ops

    ops, n, g = get_ops(), sum(lens), torch.Generator(device="cuda").manual_seed(hd + heads)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    need = [-(-(a + q) // page) for a, q in zip(starts, lens)]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(2)).tolist()
    k, v, q = rand(sum(need), kv_heads, page, hd), rand(sum(need), kv_heads, page, hd), rand(n, heads * hd)
    tables = torch.full((len(lens), max(need) + 1), -1, dtype=torch.int32)
    for i, count in enumerate(need):
        tables[i, :count] = torch.tensor(order[:count])
        order = order[count:]
    tables, outs = tables.cuda(), []
    for longest in (1, max(lens)):  # (the general kernel serves steps of few rows)
        ctx, out = _Ctx(lens, starts), torch.empty(n, heads * hd, device="cuda")
        ctx.max_q_len = longest
        before = ops.launch_counts.get("paged_attention_f32_tiles", 0)
        ops.paged_attention_general(q, k, v, tables, ctx, heads, kv_heads, hd, page, hd ** -0.5, window, out)
        assert ops.launch_counts.get("paged_attention_f32_tiles", 0) - before == (1 if longest > 1 else 0)
        outs.append(out)
    ops.check_errors()
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("m,n,k", [(700, 2048, 96), (130, 70, 40), (65, 33, 19), (1, 64, 16)])
def test_products_do_not_depend_on_the_tile(m, n, k):
    """Many rows (64 a block), few (32), one: the same chain over k, equal to adding the terms one by one."""
    from inference_engine_b200.engine.workspace import Workspace
    from inference_engine_b200.kernels import get_ops

    ops, g = get_ops(), torch.Generator(device="cuda").manual_seed(m)
    x, w = torch.randn(m, k, generator=g, device="cuda"), torch.randn(n, k, generator=g, device="cuda")
    full = ops.linear(x, w, ws=Workspace("cuda"), tag="t", out_dtype=torch.float32).clone()
    for rows in {1, min(m, 5), min(m, 33)}:
        part = ops.linear(x[m - rows:].contiguous(), w, ws=Workspace("cuda"), tag="t", out_dtype=torch.float32)
        assert torch.equal(part, full[m - rows:])
    chain = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    for i in range(k):  # (a product of two 24-bit numbers is exact in 64 bits; one rounding to 32 as in a fused multiply-add)
        chain = (chain.double() + x[:, i, None].double() * w[None, :, i].double()).float()
    torch.testing.assert_close(full, chain, atol=1e-6 * k ** 0.5, rtol=1e-6)
