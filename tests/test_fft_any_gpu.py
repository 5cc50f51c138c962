"""op_V_loc + op_K and the density on boxes whose three lengths differ, every
length with a fused plan taking each direction once, against dense FFTs in
double precision; one band, an odd block, and each setting of plane_bands.

Bounds, largest difference over the largest value and 2-norm over 2-norm: about
twice the largest of the 32 boxes (density: FP64 1.4e-15 and 6.6e-16, FP32 4.5e-7
and 2.4e-7; the dense FP64 FFTs are themselves as far from extended precision
as the FP64 kernels)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96, 100, 108, 120, 125, 128]
BOXES = [(SIZES[i], SIZES[(i + 7) % 25], SIZES[(i + 13) % 25]) for i in range(25)]
BOXES += [(n, n, 20) for n in (27, 40, 64, 75, 81, 108, 120)]     # square planes, the cubes' own kernels among them


@pytest.mark.parametrize("Ns", BOXES, ids=lambda b: "x".join(map(str, b)))
def test_box(Ns):
    import torch
    import pwb200
    N1, N2, N3 = Ns
    rng = np.random.default_rng(N1 * 10007 + N2 * 101 + N3)
    f = [np.fft.fftfreq(n, 1.0 / n) for n in Ns]
    r2 = ((f[2] / N3)[:, None, None] ** 2 + (f[1] / N2)[None, :, None] ** 2 + (f[0] / N1)[None, None, :] ** 2)
    idx = np.nonzero(r2.ravel() < 0.2 ** 2)[0]
    idx = idx[rng.permutation(len(idx))][:max(1, len(idx) - 5)]        # unordered, a few columns ragged
    N = N1 * N2 * N3
    gk2 = rng.uniform(0, 1, len(idx))          # small: rounding of the transforms, not of K, is seen
    V = rng.standard_normal(N)
    ctx = pwb200.Context(Ns, 100.0, [idx], [gk2])
    ctx.set_vloc(V)
    t = torch.from_numpy(idx).cuda()
    Vt = torch.from_numpy(V).cuda().view(N3, N2, N1)
    for dt, tol, tol2 in ((torch.complex128, 3e-15, 1.3e-15), (torch.complex64, 9e-7, 5e-7)):
        for nb, pb in ((1, 0), (5, 0), (5, 1), (5, 2), (4, 3)):
            g = torch.Generator(device="cuda").manual_seed(nb)
            x = torch.randn((nb, len(idx)), dtype=torch.complex128, device="cuda", generator=g).to(dt)
            y = torch.empty_like(x)
            ctx.set_tuning(plane_bands=pb)
            ctx.apply(0, 0, x, y, pwb200.PW_OP_K | pwb200.PW_OP_VLOC)
            c = torch.zeros((nb, N), dtype=torch.complex128, device="cuda")
            c[:, t] = x.to(torch.complex128)
            u = torch.fft.ifftn(c.view(nb, N3, N2, N1), dim=(1, 2, 3))
            ref = torch.fft.fftn(u * Vt, dim=(1, 2, 3)).reshape(nb, N)[:, t]
            ref = ref + 0.5 * torch.from_numpy(gk2).cuda() * x.to(torch.complex128)
            assert (y - ref).abs().max() <= tol * ref.abs().max(), (dt, nb, pb)
            assert torch.linalg.vector_norm(y - ref) <= tol2 * torch.linalg.vector_norm(ref), (dt, nb, pb)
            if pb:
                continue
            w = rng.uniform(0.1, 2.0, nb)
            rho = torch.zeros(N, dtype=torch.float64, device="cuda")
            ctx.calc_rhoe(0, x, w, rho)
            rr = (torch.from_numpy(w).cuda()[:, None] * (u.abs() ** 2).reshape(nb, N)).sum(dim=0) * N * N / 100.0
            assert (rho - rr).abs().max() <= tol * rr.abs().max(), (dt, nb)
            assert torch.linalg.vector_norm(rho - rr) <= tol2 * torch.linalg.vector_norm(rr), (dt, nb)
    ctx.close()
