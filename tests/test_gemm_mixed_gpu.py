"""Mixed-precision Gram and rotation at the edges of the tensor-core tiles: one
row and column, remainders of the 128-row and 32..128-column tiles and of the
32-value k-blocks, one and several splits, leading dimensions above K, and the
A^H A form that fills one triangle from the other.

Bounds per element: products of two BF16 pieces drop terms of 2^-16 of |a||b|
(A^H A keeps them), and sums round at 2^-24 per k-block; 3 2^-17 sum |a||b|
covers both sides of each complex product."""
import pytest

pytestmark = pytest.mark.gpu

REL = 3.0 * 2.0 ** -17


@pytest.fixture(scope="module")
def ctx():
    import numpy as np
    import pwb200
    from pwb200.system import Basis
    b = Basis(7.0 * np.eye(3), 4.0)
    c = pwb200.Context(b.Ns, b.CellVolume, b.idx_gw2r, b.Gk2)
    yield c
    c.check_device()
    c.close()


def block(n, K, pad, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((n, K + pad), dtype=torch.complex64, device="cuda", generator=g)[:, :K]


@pytest.mark.parametrize("K,m,n,pad", [(1, 1, 1, 0), (31, 3, 17, 1), (32, 127, 32, 0), (33, 128, 33, 3), (65, 129, 80, 0),
                                       (1009, 160, 81, 2), (5003, 257, 97, 0), (20011, 130, 161, 5), (4099, 300, 300, 0)])
def test_gram_edges(ctx, K, m, n, pad):
    import torch
    A, B = block(m, K, pad, 1), block(n, K, pad, 2)
    Ad, Bd = A.to(torch.complex128), B.to(torch.complex128)
    G0 = torch.randn((n, m), dtype=torch.complex128, device="cuda")
    ref, bound = (Ad.conj() @ Bd.T).T, REL * (Ad.abs() @ Bd.abs().T).T
    G = G0.clone()
    ctx.gram(A, B, G)
    assert ((G - ref).abs() <= bound).all()
    G.copy_(G0)
    ctx.gram(A, B, G, accumulate=True)
    assert ((G - ref - G0).abs() <= bound + 1e-15 * G0.abs()).all()
    S = torch.full((m, m), 7.0, dtype=torch.complex128, device="cuda")
    ctx.gram(A, A, S)
    refS, boundS = (Ad.conj() @ Ad.T).T, REL * (Ad.abs() @ Ad.abs().T)
    assert ((S - refS).abs() <= boundS).all()
    assert torch.equal(torch.triu(S, 1).conj(), torch.tril(S, -1).T)
    ctx.gram(A, A, S, accumulate=True)
    assert ((S - 2 * refS).abs() <= 2 * boundS).all()


@pytest.mark.parametrize("K,m,n", [(30, 5, 5), (30, 100, 100), (200, 100, 100), (80009, 3, 11), (40009, 33, 33), (9001, 256, 256),
                                   (9001, 257, 256), (3001, 480, 480)])
def test_tiles_and_parts(ctx, K, m, n):
    """Narrow and wide tiles, unsplit (one pass, both triangles of A^H A) and in
    many parts (eight lanes an element up to 65,536 of them)."""
    test_gram_edges(ctx, K, m, n, 0)


@pytest.mark.parametrize("M,n,k,pad", [(1, 1, 1, 0), (17, 3, 7, 1), (127, 32, 32, 0), (128, 33, 31, 1), (1009, 80, 65, 0),
                                       (5003, 97, 161, 3), (24001, 160, 320, 0)])
def test_rotate_edges(ctx, M, n, k, pad):
    import torch
    A = block(k, M, pad, 4)
    g = torch.Generator(device="cuda").manual_seed(5)
    U = torch.randn((n, k), dtype=torch.complex128, device="cuda", generator=g)
    X0 = block(n, M, 0, 6).contiguous()
    ref = U @ A.to(torch.complex128)
    bound = REL * (U.abs() @ A.to(torch.complex128).abs())
    X = X0.clone()
    ctx.rotate(A, U, X)
    assert ((X - ref).abs() <= bound + 2e-7 * ref.abs()).all()
    X.copy_(X0)
    ctx.rotate(A, U, X, accumulate=True)
    assert ((X - ref - X0).abs() <= bound + 4e-7 * (ref.abs() + X0.abs())).all()


@pytest.mark.parametrize("M,n,k", [(40001, 20, 33), (19001, 50, 40), (40001, 70, 5), (33333, 90, 70), (20001, 250, 100)])
def test_several_tiles_a_cta(ctx, M, n, k):
    """More output tiles than SMs, at every tile width."""
    test_rotate_edges(ctx, M, n, k, 0)


def test_several_gram_tiles_a_cta(ctx):
    test_gram_edges(ctx, 70, 1600, 1500, 1)
