"""op_V_loc + op_K and the density on boxes whose three lengths differ, every
length with a fused plan taking each direction once, against dense FFTs in
double precision; one band, an odd block, and each setting of plane_bands.

Bounds: FP64 1e-13, FP32 4e-6 of the largest value (a line of n points rounds
about log2 n times; 6 lines a value, eps 6e-8)."""
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
    gk2 = rng.uniform(0, 30, len(idx))
    V = rng.standard_normal(N)
    ctx = pwb200.Context(Ns, 100.0, [idx], [gk2])
    ctx.set_vloc(V)
    t = torch.from_numpy(idx).cuda()
    Vt = torch.from_numpy(V).cuda().view(N3, N2, N1)
    for dt, tol in ((torch.complex128, 1e-13), (torch.complex64, 4e-6)):
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
            if pb:
                continue
            w = rng.uniform(0.1, 2.0, nb)
            rho = torch.zeros(N, dtype=torch.float64, device="cuda")
            ctx.calc_rhoe(0, x, w, rho)
            rr = (torch.from_numpy(w).cuda()[:, None] * (u.abs() ** 2).reshape(nb, N)).sum(dim=0) * N * N / 100.0
            assert (rho - rr).abs().max() <= tol * rr.abs().max(), (dt, nb)
    ctx.close()
