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


@pytest.mark.parametrize("hd", [32, 64, 128])
@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("missing", [False, True])
def test_attention_does_not_look_at_hidden_values(hd, window, missing):
    """Infinities and NaN in values (and NaN in keys) of some positions reach the rows that see them and no others, which are
    the general kernel's bits; a page that the table does not hold is left out and reported, as there."""
    from inference_engine_b200.kernels import get_ops
    from inference_engine_b200.kernels.cuda_ops import KernelError

    ops, heads, kv_heads, page, lens, starts = get_ops(), 6, 2, 8, [90, 33], [50, 0]
    g = torch.Generator(device="cuda").manual_seed(hd + window)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    pages = [-(-(a + n) // page) for a, n in zip(starts, lens)]
    k, v, q = rand(sum(pages), kv_heads, page, hd), rand(sum(pages), kv_heads, page, hd), rand(sum(lens), heads * hd)
    tables = torch.full((2, max(pages)), -1, dtype=torch.int32)
    tables[0, : pages[0]] = torch.arange(pages[0])
    tables[1, : pages[1]] = torch.arange(pages[0], sum(pages))
    for at, what in ((60, "nan"), (77, "inf"), (78, "-inf"), (139, "nan")):  # (positions of the first request)
        v[at // page, :, at % page, at % 7::7] = float(what)
    v[pages[0] + 2, 1, 3, :] = float("nan")  # position 19 of the second, one of its heads
    k[100 // page, :, 100 % page, 0] = float("nan")
    if missing:
        tables[0, 3] = -1
    tables, outs = tables.cuda(), []
    for longest in (1, max(lens)):
        ctx, out = _Ctx(lens, starts), torch.empty(sum(lens), heads * hd, device="cuda")
        ctx.max_q_len = longest
        before = ops.launch_counts.get("paged_attention_f32_tiles", 0)
        ops.paged_attention_general(q, k, v, tables, ctx, heads, kv_heads, hd, page, hd ** -0.5, window, out)
        assert ops.launch_counts.get("paged_attention_f32_tiles", 0) - before == (1 if longest > 1 else 0)
        if missing:
            with pytest.raises(KernelError):
                ops.check_errors()
        else:
            ops.check_errors()
        outs.append(out)
    bad = [torch.isnan(o) for o in outs]
    assert torch.equal(*bad) and torch.equal(*(o.masked_fill(b, 0.0) for o, b in zip(outs, bad)))
    assert not bad[0][:10].any() and bad[0][10:27].any() and not bad[0][90:109].any() and bad[0][109:, heads * hd // 2:].all()


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
