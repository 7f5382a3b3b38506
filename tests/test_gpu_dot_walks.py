"""fp32 products in the reference's order over every way in which operands are staged (16-byte pieces, contiguous rows, any strides), each operand in
each of them: the same bits as for contiguous operands, at the remainders of tiles and of blocks of 32 products."""
import pytest
import torch

import jasmine_b200 as jb

pytestmark = pytest.mark.gpu


def laid_out(x, how):
    """A view with x's values: contiguous, transposed, every other element of both directions, or rows off 16-byte alignment."""
    r, c = x.shape
    if how == "rows":
        return x.contiguous()
    if how == "columns":
        return x.t().contiguous().t()
    wide = torch.full((2 * r, 2 * c + 1) if how == "strided" else (r, c + 5), torch.nan, device="cuda")
    view = wide[::2, 1::2] if how == "strided" else wide[:, 1:c + 1]
    view.copy_(x)
    return view


@pytest.mark.parametrize("M,N,K", [(1, 9, 3), (16, 16, 32), (17, 15, 33), (63, 65, 127), (65, 64, 31), (1030, 520, 70), (600, 961, 129)])
def test_same_bits_in_every_layout(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M)
    A, B = torch.randn(M, K, generator=g, device="cuda"), torch.randn(K, N, generator=g, device="cuda")
    want = jb.dot_f32(A, laid_out(B, "columns"), torch.empty(M, N, device="cuda"))  # (products contiguous in both)
    e = K * 2.0 ** -23 * (A.abs().double() @ B.abs().double())
    assert bool(((want.double() - A.double() @ B.double()).abs() <= e).all())
    for la in ("rows", "columns", "strided", "off"):
        for lb in ("rows", "columns", "strided", "off"):
            out = torch.full((M + 1, N), 7.0, device="cuda")
            jb.dot_f32(laid_out(A, la), laid_out(B, lb), out[:M])
            assert torch.equal(out[:M], want) and bool((out[M] == 7.0).all()), (la, lb)


@pytest.mark.parametrize("n,K", [(64, 64), (50, 50), (17, 17), (16, 16)])
@pytest.mark.parametrize("into", ["left", "right", "transposed"])
def test_products_of_one_tile_in_place_of_an_operand(n, K, into):
    """x <- x W of up to 64 x 64: everything is read before the first write."""
    g = torch.Generator(device="cuda").manual_seed(n)
    for _ in range(5):
        A, B = torch.randn(n, K, generator=g, device="cuda"), torch.randn(K, n, generator=g, device="cuda")
        want = jb.dot_f32(A, B, torch.empty(n, n, device="cuda"))
        out = {"left": A, "right": B, "transposed": B.t()}[into]
        jb.dot_f32(A, B, out)
        assert torch.equal(out, want)
