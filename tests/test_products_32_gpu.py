"""32-bit products put together on the tensor cores (256 of k and more) against 64 bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from inference_engine_b200.kernels import get_ops

    return get_ops("cuda")


def _product(ops, a, w):
    out = torch.full((a.shape[0], w.shape[0]), 7.0, device="cuda")
    ops.linear(a, w, out)
    return out


@pytest.mark.parametrize("k", [255, 256, 257, 300, 320, 1000, 2048])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 130])
@pytest.mark.parametrize("m", [1, 16, 17, 33, 530])
def test_error_and_rows(ops, m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m * n + k)
    a, w = (torch.randn(rows, k, generator=g, device="cuda") for rows in (m, n))
    a[:, k // 2] *= 1e4
    out = _product(ops, a, w)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    # each number's two parts leave 2^-23 of it out, the products of both second parts 2^-22, the tensor cores' sums 2^-23 each, of which
    # those of the first parts' products, two of six, count in full; then
    # ceil(k / 64) + 2 roundings.  A chain: k of them.
    bound = (9 + (k / 64 + 3) / 2) * 2 ** -23 if k >= 256 else k * 2 ** -24
    assert ((out.double() - ref).abs() <= bound * size).all()
    # a row by itself, whatever the tile: the same bits
    for row in {0, m - 1, m // 2}:
        assert torch.equal(_product(ops, a[row:row + 1].contiguous(), w), out[row:row + 1])


def test_numbers_that_are_not_finite(ops):
    """As in one chain of multiply-adds: an infinity stays one, opposite ones make no number, and a number next to the largest stays finite."""
    a, w = torch.randn(40, 320, device="cuda"), torch.randn(50, 320, device="cuda")
    a[3, 5], a[7, 9], w[11, 300], a[20, 1], a[20, 2] = float("inf"), float("nan"), float("-inf"), float("inf"), float("-inf")
    a[9] = 0
    a[9, 3] = torch.finfo(torch.float32).max
    w[:, 3] = torch.where(w[:, 3].abs() > 0.9, torch.full_like(w[:, 3], 0.9), w[:, 3])
    out, ref = _product(ops, a, w), (a.double() @ w.double().T).float()
    assert torch.equal(out.isnan(), ref.isnan()) and torch.equal(out.isinf(), ref.isinf())
    assert torch.equal(out[out.isinf()], ref[ref.isinf()])
    finite = ref.isfinite()
    torch.testing.assert_close(out[finite], ref[finite], rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("rows,columns,k", [(5, 300, 256), (64, 70, 1001), (377, 1024, 1024)])
@pytest.mark.parametrize("weight", ["one", "any"])
def test_products_of_a_single_term(ops, rows, columns, k, weight):
    """A matrix that selects (one entry a row that is not 0).  Of an operand's two parts of 11 bits the second one, up to 2^-11 of it, loses its last bit,
    2^-23 of the operand; the product of both second parts, up to 2^-22 of the result, is left out; and the tensor cores cut off where they add
    the first parts' product to the rest, up to 2^-22.  With a weight of 1, which has no second part, the first of these is all.  (Below 256 of k a chain
    of multiply-adds rounds such a product once: 2^-24, and 0 with a weight of 1.)"""
    g = torch.Generator(device="cuda").manual_seed(k)
    at = torch.randint(0, k, (columns,), generator=g, device="cuda")
    w = torch.zeros(columns, k, device="cuda")
    w[torch.arange(columns, device="cuda"), at] = 1.0 if weight == "one" else torch.randn(columns, generator=g, device="cuda")
    a = torch.randn(rows, k, generator=g, device="cuda")
    want = a.double()[:, at] * w.double().sum(dim=1)
    error = ((_product(ops, a, w).double() - want) / want).abs().max()
    assert error <= (1 if weight == "one" else 6) * 2.0 ** -23
