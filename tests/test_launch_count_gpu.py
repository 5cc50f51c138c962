"""pw_launch_count against what was launched: op_H, Gram and rotation recorded into
a CUDA graph whose kernel nodes are counted, at sizes with one and with several
parts of the sum; the eigensolver's by its steps."""
import numpy as np
import pytest

from conftest import cuda_ok

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fcc():
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import pwb200
    from oracle import systems
    H = systems.Ham_Si_fcc(meshk=(1, 1, 1), extra_states=4)
    ctx = pwb200.Context(H.pw.Ns, H.pw.CellVolume, H.pw.gvecw.idx_gw2r, [H.pw.Gk2(0)])
    ctx.set_vloc(H.V_Ps_loc)
    ctx.set_nonlocal(0, H.betaNL[0])
    ctx.set_nonlocal_coef(H.nl_triplets)
    yield ctx, H.pw.gvecw.Ngw[0]
    ctx.close()


def recorded(ctx, call):
    """(kernel nodes of the recorded call, the counter's difference)"""
    import torch
    from cuda.bindings import runtime as rt
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        call()                                    # workspaces
        s.synchronize()
        assert rt.cudaStreamBeginCapture(s.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed)[0] == 0
        n0 = ctx.launch_count()
        try:
            call()
        finally:
            err, graph = rt.cudaStreamEndCapture(s.cuda_stream)
    n1 = ctx.launch_count()
    assert err == 0
    _, _, n = rt.cudaGraphGetNodes(graph)
    err, nodes, n = rt.cudaGraphGetNodes(graph, n)
    kinds = [rt.cudaGraphNodeGetType(v)[1] for v in nodes[:n]]
    rt.cudaGraphDestroy(graph)
    return sum(k == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds), n1 - n0


@pytest.mark.parametrize("prec", ["c128", "c64"])
def test_recorded_calls(fcc, prec):
    import torch
    import pwb200
    ctx, ngw = fcc
    dt = torch.complex128 if prec == "c128" else torch.complex64

    def r(*shape, d=dt):
        return torch.randn(shape, dtype=d, device="cuda")
    for nb in (1, 8, 40):
        x, y = r(nb, ngw), r(nb, ngw)
        for ops in (pwb200.PW_OP_H, pwb200.PW_OP_VNL, pwb200.PW_OP_K, pwb200.PW_OP_VLOC | pwb200.PW_ACCUMULATE):
            a, b = recorded(ctx, lambda: ctx.apply(0, 0, x, y, ops))
            assert a == b, (nb, ops)
    for K, m in ((20, 8), (50, 33), (3000, 8), (700, 300)):
        A, B = r(m, K), r(m, K)
        C, U, X = r(m, m, d=torch.complex128), r(m, m, d=torch.complex128), r(m, K)
        for f in (lambda: ctx.gram(A, B, C), lambda: ctx.gram(A, A, C), lambda: ctx.rotate(A, U, X)):
            a, b = recorded(ctx, f)
            assert a == b, (K, m)


def test_eigensolver_steps(fcc):
    import torch
    ctx, _ = fcc
    for n, grid in ((40, 0), (300, 1), (1100, 1)):
        for G in (False, True):
            for vectors in (False, True):
                A = torch.randn((n, n), dtype=torch.complex128, device="cuda")
                T, E = A + A.conj().T, torch.eye(n, dtype=torch.complex128, device="cuda")
                n0 = ctx.launch_count()
                ctx.eigh(T, E if G else None, k=3, vectors=vectors)
                # Hermitian T; with G its own, Cholesky, two products, two transposes;
                # tridiagonal form, its check, the values; vectors, back (and by L^-H)
                want = 1 + 6 * G + grid + 1 + 2 + (2 + G) * vectors
                assert ctx.launch_count() - n0 == want, (n, G, vectors)
