"""The FP64 eigensolver at the edges of its blocks: orders around one and two
32-column panels, one to four eigenvectors per CTA of the back-transformation,
and spectra with exact zeros off the diagonal, repeated eigenvalues and
unusual norms.  Bounds: 64 n eps of the norm for residuals and eigenvalues,
1e-9 for orthogonality inside clusters (as the solver's own 1e-7 threshold)."""
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


def dev(A):
    import torch
    return torch.from_numpy(np.ascontiguousarray(A.T)).cuda()


def check(ctx, T, k, G=None):
    n = T.shape[0]
    lam, S = ctx.eigh(dev(T), None if G is None else dev(G), k=k)
    lam, S = lam.cpu().numpy(), S.cpu().numpy().T
    nrm = np.abs(np.linalg.norm(T, 2)) if n > 1 else max(abs(T[0, 0]), 1e-300)
    B = np.eye(n) if G is None else G
    # the zero matrix's search interval is +-1e-300 wide
    tol = 64 * n * EPS * nrm * (1.0 if G is None else np.linalg.cond(G)) + 1e-299
    ref = np.linalg.eigvalsh(T) if G is None else None
    if ref is not None:
        assert np.abs(lam - ref[:k]).max() <= tol
    assert np.abs(T @ S - (B @ S) * lam).max() <= tol
    assert np.abs(S.conj().T @ B @ S - np.eye(k)).max() < 1e-9
    assert (np.diff(lam) >= -tol).all()


def herm(n, seed):
    r = np.random.default_rng(seed)
    A = r.standard_normal((n, n)) + 1j * r.standard_normal((n, n))
    return A + A.conj().T


@pytest.mark.parametrize("n,k", [(1, 1), (2, 2), (3, 1), (31, 31), (32, 7), (33, 33), (34, 5), (64, 64), (65, 20),
                                 (97, 33), (130, 130), (257, 85), (300, 297), (481, 160), (513, 171), (600, 595), (700, 3)])
def test_orders(ctx, n, k):
    check(ctx, herm(n, n), k)


@pytest.mark.parametrize("n,k", [(16, 16), (17, 3), (255, 80), (256, 256), (258, 70), (512, 40), (1024, 9), (1025, 9)])
def test_last_columns_in_one_cluster(ctx, n, k):
    """The last 256 columns of the tridiagonalisation go to one cluster, those
    before them to the grid (registers up to 1024, L2 above)."""
    check(ctx, herm(n, n), k)


@pytest.mark.parametrize("n,want", [(1, 2), (256, 2), (257, 3), (480, 3), (512, 3), (513, 3), (700, 3), (1024, 3), (1025, 2)])
def test_kernels_of_the_tridiagonalisation(n, want):
    """On a whole B200: the register kernel (1) for the columns before the last 256
    up to n = 1024, the cluster (2) for those."""
    import ctypes as C
    import pwb200
    f = pwb200.lib().pwk_test_tri_route
    f.restype, f.argtypes = C.c_int, [C.c_int, C.c_int]
    assert f(0, n) == want


@pytest.mark.parametrize("n,k", [(1, 1), (33, 11), (100, 100), (480, 160), (545, 300)])
def test_generalized(ctx, n, k):
    r = np.random.default_rng(n + 1)
    B = r.standard_normal((n, n)) + 1j * r.standard_normal((n, n))
    check(ctx, herm(n, n), k, np.eye(n) + 0.1 / np.sqrt(n) * (B + B.conj().T))


@pytest.mark.parametrize("scale", [1e-12, 1.0, 1e6])
def test_structured_spectra(ctx, scale):
    n = 70
    check(ctx, scale * np.diag(np.arange(n, dtype=float) - 20).astype(complex), n)          # no coupling at all
    check(ctx, scale * np.eye(n, dtype=complex), 9)                                          # one eigenvalue
    blocks = np.kron(np.eye(n // 2), np.array([[1.0, 2.0], [2.0, 1.0]])).astype(complex)     # two, decoupled
    check(ctx, scale * blocks, n // 2)
    Q, _ = np.linalg.qr(herm(n, 5))
    check(ctx, scale * (Q * np.repeat(np.arange(n // 7), 7)) @ Q.conj().T, 30)               # sevenfold levels
    T = np.zeros((n, n), dtype=complex)
    check(ctx, T, 4)
