"""FP64 Gram and rotation at the edges of the tensor-core tiles: one column,
remainders of the 8-wide blocks and of the 32..80-wide tiles, K below and
above one 8-step, K that splits unevenly, leading dimensions above K, and the
A^H A form that fills one triangle from the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.2e-16


@pytest.fixture(scope="module")
def ctx():
    import pwb200
    from pwb200.system import Basis
    b = Basis(7.0 * np.eye(3), 4.0)
    c = pwb200.Context(b.Ns, b.CellVolume, b.idx_gw2r, b.Gk2)
    yield c
    c.close()


def block(n, K, pad, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((n, K + pad), dtype=torch.complex128, device="cuda", generator=g)[:, :K]


@pytest.mark.parametrize("K,m,n,pad", [(1, 1, 1, 0), (7, 3, 17, 5), (8, 16, 16, 0), (9, 33, 31, 1), (63, 47, 49, 0),
                                       (65, 80, 81, 3), (1009, 64, 5, 0), (5003, 113, 97, 2), (20011, 240, 161, 0)])
def test_gram_edges(ctx, K, m, n, pad):
    """|error| <= 2 K eps sum |a||b| per element (K products and sums, each
    within eps, in any order; the factor 2 for the four real products)."""
    import torch
    A, B = block(m, K, pad, 1), block(n, K, pad, 2)
    G0 = block(n, m, 0, 3).clone()
    bound = 2 * K * EPS * (A.abs() @ B.abs().T).T + 4 * EPS
    ref = (A.conj() @ B.T).T
    G = G0.clone()
    ctx.gram(A, B, G)
    assert ((G - ref).abs() <= bound).all()
    G.copy_(G0)
    ctx.gram(A, B, G, accumulate=True)
    assert ((G - ref - G0).abs() <= bound + 4 * EPS * G0.abs()).all()
    S = torch.full((m, m), 7.0, dtype=torch.complex128, device="cuda")
    ctx.gram(A, A, S)
    refS = (A.conj() @ A.T).T
    assert ((S - refS).abs() <= 2 * K * EPS * (A.abs() @ A.abs().T) + 4 * EPS).all()
    assert torch.equal(torch.triu(S, 1).conj(), torch.tril(S, -1).T)
    ctx.gram(A, A, S, accumulate=True)
    assert ((S - 2 * refS).abs() <= 4 * K * EPS * (A.abs() @ A.abs().T) + 8 * EPS).all()


@pytest.mark.parametrize("K,m,n", [(30, 5, 5), (24007, 1, 1), (24007, 3, 11), (40009, 33, 33), (9001, 256, 256),
                                   (9001, 257, 256)])
def test_few_values_in_many_parts(ctx, K, m, n):
    """Sums without parts, with one thread and with eight lanes an element (up to
    65,536 elements), both triangles; bound as above."""
    test_gram_edges(ctx, K, m, n, 0)


@pytest.mark.parametrize("M,n,k,pad", [(1, 1, 1, 0), (17, 3, 7, 1), (63, 16, 8, 0), (65, 33, 9, 2), (1009, 48, 50, 0),
                                       (5003, 81, 161, 3), (12007, 161, 480, 0)])
def test_rotate_edges(ctx, M, n, k, pad):
    import torch
    A, U = block(k, M, pad, 4), block(n, k, 0, 5).contiguous()
    X0 = block(n, M, 0, 6).clone()
    ref = U @ A
    bound = 2 * k * EPS * (U.abs() @ A.abs()) + 4 * EPS
    X = X0.clone()
    ctx.rotate(A, U, X)
    assert ((X - ref).abs() <= bound).all()
    X.copy_(X0)
    ctx.rotate(A, U, X, accumulate=True)
    assert ((X - ref - X0).abs() <= bound + 4 * EPS * X0.abs()).all()


@pytest.mark.parametrize("K,m", [(700, 36), (24000, 60), (24000, 180)])
def test_long_sums_against_extended_precision(ctx, K, m):
    """Rows of falling weight, as wavefunctions: 2-norm error of 24 x 24 values of A^H B
    and of a rotation, at most 8e-16, about twice the measured 2e-16 to 5e-16 (sums that
    every product rounds: 1.6e-15 and 5.0e-15 over 24,000)."""
    import torch
    w = 1.0 / (1.0 + 30.0 * (torch.arange(K, device="cuda", dtype=torch.float64) / K) ** (2.0 / 3.0))
    A, B = block(m, K, 0, 11) * w, block(m, K, 0, 12) * w
    G = torch.empty((m, m), dtype=torch.complex128, device="cuda")
    ctx.gram(A, B, G)
    a, b = (x[:24].cpu().numpy().astype(np.clongdouble) for x in (A, B))
    ref, got = (a.conj() @ b.T).T, G[:24, :24].cpu().numpy()
    assert np.sqrt((np.abs(got - ref) ** 2).sum() / (np.abs(ref) ** 2).sum()) < 8e-16
    U, X = block(24, m, 0, 13).contiguous(), torch.empty((24, K), dtype=torch.complex128, device="cuda")
    ctx.rotate(A, U, X)
    ref = U.cpu().numpy().astype(np.clongdouble) @ A[:, :50].cpu().numpy().astype(np.clongdouble)
    got = X[:, :50].cpu().numpy()
    assert np.sqrt((np.abs(got - ref) ** 2).sum() / (np.abs(ref) ** 2).sum()) < 4e-16
