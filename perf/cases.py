"""The work that users of pwb200 have it do, as cases that can be timed.

A case is one call (or the few calls that always go together) of the public
host package on inputs like those of a plane-wave DFT run: bulk silicon in
conventional cubic cells repeated nx x ny x nz times (a = 10.2631 bohr, atoms
displaced by up to 0.02 bohr), its two-atom fcc cell, and fcc aluminium with
a k-mesh; GTH pseudopotentials; cutoffs from 8 to 15 Ha.

kinds
  opH     op_H (K + V_loc + V_Ps_nloc) on a block of bands at one k-point:
          the inner call of every eigensolver and of direct minimisation
  host    the same through the drop-in for host arrays (pinned ComplexF64)
  rhoe    calc_rhoe of the occupied bands, once per SCF iteration
  rr      the Rayleigh-Ritz products of LOBPCG: Q'HQ, Q'Q and Q U
  eigh    the reduced generalized eigenproblem of an eigensolver iteration
  multik  op_H over all k-points in one call
  lobpcg  a fixed number of LOBPCG iterations and the density of the result:
          the diagonalisation step of an SCF iteration
"""
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "pwdft.jl_b200"))

import pwb200  # noqa: E402
from pwb200.system import Basis, GTH, System, kpoint_grid, projector_table  # noqa: E402

A_SI, A_AL = 10.2631, 7.6524
DIAMOND = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0],
                    [.25, .25, .25], [.25, .75, .75], [.75, .25, .75], [.75, .75, .25]])
FCC = DIAMOND[:4]
# GTH-LDA parameters, for the potentials and the 64-bit results below
SI = {"z": 4.0, "rloc": 0.44, "c1": -7.33610297, "r": (0.42273813, 0.48427842),
      "h0": ((5.90692831, -1.26189397), (-1.26189397, 3.25819622)), "h1": 2.72701346, "file": "Si-q4.gth"}
AL = {"z": 3.0, "rloc": 0.45, "c1": -8.49135116, "r": (0.46010427, 0.53674439),
      "h0": ((5.08833953, -1.03784325), (-1.03784325, 2.67969975)), "h1": 2.19343827, "file": "Al-q3.gth"}


def listed():
    return [
        # the reference's own test system (two atoms, 27^3 grid), one k-point
        # off Gamma: what counts is latency
        dict(name="opH_si2_fp64", kind="opH", lat="fcc", nx=1, ny=1, nz=1, ecut=15.0, kshift=0.25, bands=8, dtype="fp64"),
        # the conventional cell, on a grid (40^3) that no benchmark uses
        dict(name="opH_si8_mixed", kind="opH", lat="sc", nx=1, ny=1, nz=1, ecut=15.0, kshift=0.0, bands=20, dtype="mixed"),
        # a flat supercell (75 x 75 x 40), an odd block, in the reference's precision
        dict(name="opH_si32_slab_fp64", kind="opH", lat="sc", nx=2, ny=2, nz=1, ecut=15.0, kshift=0.0, bands=81, dtype="fp64"),
        # the benchmark's op_H: 64 atoms, 160 bands
        dict(name="opH_si64_mixed", kind="opH", lat="sc", nx=2, ny=2, nz=2, ecut=15.0, kshift=0.0, bands=160, dtype="mixed"),
        # the largest system of the benchmark: 216 atoms, 480 bands
        dict(name="opH_si216_mixed", kind="opH", lat="sc", nx=3, ny=3, nz=3, ecut=15.0, kshift=0.0, bands=480, dtype="mixed"),
        # a host program handing over its ComplexF64 arrays
        dict(name="host_si64_fp64", kind="host", lat="sc", nx=2, ny=2, nz=2, ecut=15.0, kshift=0.0, bands=160, dtype="fp64"),
        # density of the 128 occupied bands of 64 atoms
        dict(name="rhoe_si64_fp64", kind="rhoe", lat="sc", nx=2, ny=2, nz=2, ecut=15.0, kshift=0.0, bands=128, dtype="fp64"),
        # Rayleigh-Ritz products of 160 bands (64 atoms), reference precision
        dict(name="rr_160_fp64", kind="rr", K=23871, bands=160, dtype="fp64"),
        # and of 480 bands (216 atoms) on the mixed path
        dict(name="rr_480_mixed", kind="rr", K=80797, bands=480, dtype="mixed"),
        # the reduced eigenproblem that goes with 160 bands
        dict(name="eigh_480", kind="eigh", n=480, k=160),
        # all k-points of a small metal in one call (8 x 8 x 8 mesh, 10 bands each)
        dict(name="multik_al4_mixed", kind="multik", mesh=8, ecut=15.0, bands=10, dtype="mixed"),
        # the diagonalisation of one SCF iteration: 4 LOBPCG iterations and the density
        dict(name="lobpcg_si64_mixed", kind="lobpcg", lat="sc", nx=2, ny=2, nz=2, ecut=15.0, kshift=0.0, bands=160,
             iters=4, dtype="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["opH", "opH", "opH", "opH", "host", "rhoe", "rhoe", "rr", "rr", "eigh", "multik", "lobpcg"])
    if kind == "rr":
        nb = _log(rng, 4, 480)
        return dict(kind="rr", K=_log(rng, 3 * nb + 50, 80000), bands=nb, dtype=rng.choice(["fp64", "mixed"]))\
            if nb <= 200 else dict(kind="rr", K=_log(rng, 3 * nb + 50, 80000), bands=nb, dtype="mixed")
    if kind == "eigh":
        n = _log(rng, 12, 900)
        return dict(kind="eigh", n=n, k=max(1, n // 3))
    if kind == "multik":
        return dict(kind="multik", mesh=rng.randint(2, 7), ecut=15.0, bands=rng.randint(4, 13),
                    dtype=rng.choice(["fp64", "mixed"]))
    dtype = rng.choice(["fp64", "mixed"])
    ecut = round(rng.uniform(8.0, 15.0), 1)
    if kind in ("opH", "rhoe") and rng.random() < 0.2:
        return dict(kind=kind, lat="fcc", nx=1, ny=1, nz=1, ecut=ecut, kshift=rng.choice([0.0, 0.125, 0.25]),
                    bands=rng.randint(1, 12), dtype=dtype)
    top = 2 if kind in ("host", "lobpcg") else 3
    while True:
        nx, ny, nz = (rng.randint(1, top) for _ in range(3))
        if nx * ny * nz <= 12:
            break
    most = 20 * nx * ny * nz                       # 2.5 bands an atom, as the benchmark has
    bands = _log(rng, max(1, most // 16), most)
    if kind == "lobpcg":
        bands = max(4, min(bands, 120))
    c = dict(kind=kind, lat="sc", nx=nx, ny=ny, nz=nz, ecut=ecut, kshift=0.0, bands=bands, dtype=dtype)
    if kind == "lobpcg":
        c["iters"] = rng.randint(2, 4)
    return c


# ------------------------------------------------------------------ inputs
def _lattice(lat, nx, ny, nz):
    if lat == "fcc":
        LL = 0.5 * A_SI * np.array([[-1., 0, -1], [0, 1, 1], [1, 1, 0]])
        frac = np.array([[0, 0, 0], [.25, .25, .25]])
    elif lat == "al4":
        LL, frac = A_AL * np.eye(3), FCC
    else:
        LL = A_SI * np.diag([float(nx), float(ny), float(nz)])
        frac = np.array([(b + np.array([i, j, k])) / np.array([nx, ny, nz])
                         for i in range(nx) for j in range(ny) for k in range(nz) for b in DIAMOND])
    return LL, (LL @ frac.T)


@functools.lru_cache(maxsize=32)
def _basis(lat, nx, ny, nz, ecut, kshift, mesh):
    LL, _ = _lattice(lat, nx, ny, nz)
    if mesh:
        kpts, wk = kpoint_grid(LL, (mesh, mesh, mesh))
    else:
        kpts, wk = 2 * np.pi * np.linalg.inv(LL.T) @ (kshift * np.ones((3, 1))), np.ones(1)
    b = Basis(LL, ecut, kpts=kpts)
    gk = [b.G[b.idx_gw2g[i]] + b.kpts[:, i][None, :] for i in range(b.Nkpt)]
    return b, gk, wk


def _of(case):
    if case["kind"] == "multik":
        return "al4", 1, 1, 1, float(case["ecut"]), 0.0, int(case["mesh"])
    return case["lat"], case["nx"], case["ny"], case["nz"], float(case["ecut"]), float(case["kshift"]), 0


def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + salt)


def _positions(case, seed):
    _, pos = _lattice(*_of(case)[:4])
    return pos + np.random.default_rng(int(seed)).uniform(-0.02, 0.02, pos.shape)


def _vloc(psp, b, pos):
    """The GTH local potential of the atoms plus the smooth part that Hartree
    and exchange-correlation add (here a Gaussian of each atom's density)."""
    G, G2 = torch.from_numpy(b.G).cuda(), torch.from_numpy(b.G2).cuda()
    sf = torch.zeros(b.Ng, dtype=torch.complex128, device="cuda")
    for a in range(pos.shape[1]):
        sf += torch.exp(-1j * (G @ torch.from_numpy(pos[:, a].copy()).cuda()))
    x = G2 * psp["rloc"] ** 2
    e = torch.exp(-0.5 * x)
    safe = torch.where(G2 > 1e-12, G2, torch.ones_like(G2))
    v = -4 * math.pi * psp["z"] / safe * e + math.sqrt(8 * math.pi ** 3) * psp["rloc"] ** 3 * e * psp["c1"]
    v = v + 4 * math.pi * psp["z"] / safe * torch.exp(-G2)
    v = torch.where(G2 > 1e-12, v, torch.zeros_like(v))
    grid = torch.zeros(b.Npoints, dtype=torch.complex128, device="cuda")
    grid[torch.from_numpy(b.idx_g2r).cuda()] = sf * v / b.CellVolume
    N1, N2, N3 = b.Ns
    return (torch.fft.ifftn(grid.view(N3, N2, N1)).real * b.Npoints).reshape(-1).contiguous()


def _block(nb, gk2, seed, salt, dtype):
    """nb orthonormal bands whose coefficients fall off with the kinetic energy."""
    ngw = len(gk2)
    x = torch.randn((nb, ngw), dtype=torch.complex128, device="cuda", generator=_gen(seed, salt))
    x = x / (1.0 + torch.from_numpy(gk2).cuda())
    L = torch.linalg.cholesky(x.conj() @ x.T)                 # x x^H of the bands
    x = torch.linalg.solve_triangular(L.conj(), x, upper=False)
    return x.to(torch.complex64 if dtype == "mixed" else torch.complex128).contiguous()


def _context(case, seed):
    """The context a program keeps for its geometry: basis, V_loc, projectors."""
    b, gk, wk = _basis(*_of(case))
    psp = AL if case["kind"] == "multik" else SI
    pos = _positions(case, seed)
    LL, _ = _lattice(*_of(case)[:4])
    ctx = pwb200.Context(b.Ns, b.CellVolume, b.idx_gw2r, b.Gk2)
    V = _vloc(psp, b, pos)
    ctx.set_vloc_device(V)
    sysm = System(["Al" if psp is AL else "Si"] * pos.shape[1], pos, LL)
    pspots = [GTH(os.path.join(ROOT, "tests", "golden", "psp", psp["file"]))]
    table, trip = projector_table(sysm, b, pspots)
    for ik in range(b.Nkpt):
        ctx.set_gkvec(ik, gk[ik])
        ctx.build_nonlocal(ik, table, pos)
    ctx.set_nonlocal_coef(trip)
    return ctx, b, V


def _weights(nb):
    return np.full(nb, 2.0)


def _rr_inputs(case, seed):
    K, nb = case["K"], case["bands"]
    dt = torch.complex64 if case["dtype"] == "mixed" else torch.complex128
    g = _gen(seed, 3)
    decay = 1.0 / (1.0 + 30.0 * (torch.arange(K, device="cuda", dtype=torch.float64) / K) ** (2.0 / 3.0))

    def block(n):
        out = torch.empty((n, K), dtype=dt, device="cuda")
        for j in range(0, n, 160):
            x = torch.randn((min(160, n - j), K), dtype=torch.complex128, device="cuda", generator=g) * decay
            out[j:j + 160] = x / torch.linalg.vector_norm(x, dim=1, keepdim=True)
        return out
    Q, HQ = block(3 * nb), block(3 * nb)
    U, _ = torch.linalg.qr(torch.randn((3 * nb, nb), dtype=torch.complex128, device="cuda", generator=g))
    return Q, HQ, U.T.contiguous()


def _eigh_inputs(case, seed):
    """T and G as a Rayleigh-Ritz step forms them: Ritz values from -0.3 to
    10 Ha plus coupling, an overlap near the unit matrix."""
    n = case["n"]
    g = _gen(seed, 4)
    A = torch.randn((n, n), dtype=torch.complex128, device="cuda", generator=g)
    B = torch.randn((n, n), dtype=torch.complex128, device="cuda", generator=g)
    d = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    T = torch.diag(-0.3 + 10.3 * d * d).to(torch.complex128) + 0.05 / math.sqrt(n) * (A + A.conj().T)
    G = torch.eye(n, dtype=torch.complex128, device="cuda") + 0.1 / math.sqrt(n) * (B + B.conj().T)
    return T.contiguous(), G.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("rr", "eigh"):
        b, _, _ = _basis("fcc", 1, 1, 1, 8.0, 0.0, 0)
        s = {"kind": kind, "ctx": pwb200.Context(b.Ns, b.CellVolume, b.idx_gw2r, b.Gk2)}
        if kind == "eigh":
            s["T"], s["G"] = _eigh_inputs(case, seed)
            s["k"] = case["k"]
            return s
        s["Q"], s["HQ"], s["U"] = _rr_inputs(case, seed)
        m = 3 * case["bands"]
        s["T"] = torch.empty((m, m), dtype=torch.complex128, device="cuda")
        s["G"] = torch.empty_like(s["T"])
        s["X"] = torch.empty((case["bands"], case["K"]), dtype=s["Q"].dtype, device="cuda")
        return s
    ctx, b, _ = _context(case, seed)
    s = {"kind": kind, "ctx": ctx}
    if kind == "multik":
        nb, dt = case["bands"], torch.complex64 if case["dtype"] == "mixed" else torch.complex128
        s["iks"] = list(range(b.Nkpt))
        flat = torch.empty(nb * sum(b.Ngw), dtype=dt, device="cuda")
        s["out"] = torch.empty_like(flat)
        s["psi"], s["Hpsi"], o = [], [], 0
        for ik in s["iks"]:
            n = nb * b.Ngw[ik]
            s["psi"].append(flat[o:o + n].view(nb, b.Ngw[ik]))
            s["Hpsi"].append(s["out"][o:o + n].view(nb, b.Ngw[ik]))
            s["psi"][ik].copy_(_block(nb, b.Gk2[ik], seed, 10 + ik, case["dtype"]))
            o += n
        return s
    psi = _block(case["bands"], b.Gk2[0], seed, 1, "fp64" if kind == "host" else case["dtype"])
    if kind == "host":
        # pinned arrays of the reference's layout, (Ngw, bands) in Fortran order
        s["dtype"] = pwb200.PW_C64 if case["dtype"] == "mixed" else pwb200.PW_C128
        s["pin"] = [torch.empty(psi.shape, dtype=torch.complex128, pin_memory=True) for _ in range(2)]
        s["pin"][0].copy_(psi)
        s["psi"], s["Hpsi"] = (p.numpy().T for p in s["pin"])
        return s
    s["psi"] = psi
    if kind == "opH":
        s["Hpsi"] = torch.empty_like(psi)
    else:
        s["rho"] = torch.empty(b.Npoints, dtype=torch.float64, device="cuda")
        s["w"] = _weights(case["bands"])
        s["iters"] = case.get("iters")
    return s


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "opH":
        ctx.apply(0, 0, s["psi"], s["Hpsi"])
        return s["Hpsi"]
    if kind == "host":
        return ctx.op_H_host(0, 0, s["psi"], s["Hpsi"], dtype=s["dtype"])
    if kind == "rhoe":
        ctx.calc_rhoe(0, s["psi"], s["w"], s["rho"])
        return s["rho"]
    if kind == "rr":
        ctx.gram(s["Q"], s["HQ"], s["T"])
        ctx.gram(s["Q"], s["Q"], s["G"])
        ctx.rotate(s["Q"], s["U"], s["X"])
        return {"T": s["T"], "G": s["G"], "X": s["X"]}
    if kind == "eigh":
        lam, S = ctx.eigh(s["T"].clone(), s["G"].clone(), k=s["k"])     # both are overwritten
        return {"lam": lam, "P": S.T @ S.conj()}                        # S up to phases: S S^H
    if kind == "multik":
        ctx.apply_multi(s["iks"], 0, s["psi"], s["Hpsi"])
        return s["out"]
    X = s["psi"].clone()                                                # the start is overwritten
    ev, _ = ctx.lobpcg(0, 0, X, tol=0.0, nitermax=s["iters"])
    ctx.calc_rhoe(0, X, s["w"], s["rho"])
    return {"evals": ev, "rho": s["rho"]}


# ------------------------------------------------------- what cannot be saved
@functools.lru_cache(maxsize=256)
def _columns(key, ik):
    b, _, _ = _basis(*key)
    idx, (N1, N2, N3) = b.idx_gw2r[ik], b.Ns
    return len(np.unique(idx % (N1 * N2))), len(np.unique(idx % N1))


def _fft_flops(key, ik):
    """One 3-D transform of a band, from the columns that hold a plane wave
    to all points: 5 n log2 n for a line of n."""
    b, _, _ = _basis(*key)
    N1, N2, N3 = b.Ns
    ncol, nxa = _columns(key, ik)
    return 5.0 * (ncol * N3 * math.log2(N3) + nxa * N3 * N2 * math.log2(N2) + N2 * N3 * N1 * math.log2(N1))


def _op_work(key, ik, nb, c):
    b, _, _ = _basis(*key)
    nbeta = 5 * _lattice(*key[:4])[1].shape[1]
    ngw = b.Ngw[ik]
    return {"bytes": c * ngw * (2.0 * nb + nbeta), "flops": nb * (2 * _fft_flops(key, ik) + 16.0 * nbeta * ngw)}


def work(case):
    kind = case["kind"]
    c = 8.0 if case.get("dtype") == "mixed" else 16.0
    if kind == "rr":
        K, nb = float(case["K"]), case["bands"]
        m = 3 * nb
        return {"bytes": c * K * (2 * m + nb) + 16.0 * (2 * m * m + m * nb),
                "flops": 8.0 * K * (m * m + m * m / 2.0 + m * nb)}    # Q'Q is Hermitian: one half
    if kind == "eigh":
        n, k = float(case["n"]), case["k"]
        # Cholesky, two-sided reduction, tridiagonal form, vectors back
        return {"bytes": 16.0 * (2 * n * n + n * n) + 8 * k, "flops": n ** 3 * (4 / 3 + 4 + 16 / 3) + 12.0 * n * n * k}
    key = _of(case)
    b, _, _ = _basis(*key)
    nb = case["bands"]
    if kind == "multik":
        ws = [_op_work(key, ik, nb, c) for ik in range(b.Nkpt)]
        return {"bytes": c / 2 * b.Npoints + sum(w["bytes"] for w in ws), "flops": sum(w["flops"] for w in ws)}
    w = _op_work(key, 0, nb, c)
    if kind in ("opH", "host"):
        io = 16.0 if kind == "host" else c
        return {"bytes": w["bytes"] + c / 2 * b.Npoints + (io - c) * 2 * nb * b.Ngw[0], "flops": w["flops"]}
    rho = {"bytes": c * b.Ngw[0] * nb + 8.0 * b.Npoints, "flops": nb * (_fft_flops(key, 0) + 3.0 * b.Npoints)}
    if kind == "rhoe":
        return rho
    ngw, m, it = float(b.Ngw[0]), 3 * nb, case["iters"]
    # each iteration: op_H, X'HX, the residual, W'W and P'P, Q'HQ and Q'Q
    # (Hermitian: one half each), X, HX, P and HP from Q and HQ
    gemm = 8.0 * ngw * (nb * nb / 2 + nb * nb + nb * nb + m * m + 2 * m * nb + 4 * nb * nb)
    eig = work({"kind": "eigh", "n": m, "k": nb})["flops"]
    return {"bytes": w["bytes"] + c / 2 * b.Npoints + rho["bytes"],
            "flops": (it + 1) * w["flops"] + it * (gemm + eig) + rho["flops"]}


# ------------------------------------------------------- results in 64 bits
class _Op:
    """op_H of one k-point in plain torch: dense FFTs, dense projectors."""

    def __init__(self, case, seed, ik=0):
        key = _of(case)
        b, gk, _ = _basis(*key)
        psp = AL if case["kind"] == "multik" else SI
        pos = _positions(case, seed)
        self.b, self.V = b, _vloc(psp, b, pos)
        self.set_k(ik, psp, pos, gk[ik])

    def set_k(self, ik, psp, pos, gk):
        b = self.b
        self.idx = torch.from_numpy(b.idx_gw2r[ik]).cuda()
        self.gk2 = torch.from_numpy(b.Gk2[ik]).cuda()
        g = torch.from_numpy(np.ascontiguousarray(gk)).cuda()
        g2 = (g * g).sum(dim=1)
        r0, r1 = psp["r"]

        def pref(lq, r):
            return 4.0 * math.pi ** 1.25 * math.sqrt(2.0 ** (lq + 1) * r ** (2 * lq + 3) / b.CellVolume)
        x0, x1 = g2 * r0 * r0, g2 * r1 * r1
        y0, y1 = 0.5 / math.sqrt(math.pi), math.sqrt(0.75 / math.pi)
        s1 = pref(0, r0) * torch.exp(-0.5 * x0) * y0
        s2 = s1 * (3.0 - x0) * 2.0 / math.sqrt(15.0)
        p = (pref(1, r1) * torch.exp(-0.5 * x1) / math.sqrt(3.0) * y1)[None, :] * g.T
        self.radial = torch.cat([s1[None], s2[None], p]).to(torch.complex128)             # (5, Ngw)
        D = torch.zeros((5, 5), dtype=torch.complex128, device="cuda")
        D[:2, :2] = torch.tensor(psp["h0"], dtype=torch.complex128)
        for i in range(2, 5):
            D[i, i] = psp["h1"]
        self.D, self.g, self.pos = D, g, torch.from_numpy(pos.copy()).cuda()

    def grid(self, x):
        N1, N2, N3 = self.b.Ns
        f = torch.zeros((x.shape[0], self.b.Npoints), dtype=torch.complex128, device="cuda")
        f[:, self.idx] = x
        return torch.fft.ifftn(f.view(-1, N3, N2, N1), dim=(1, 2, 3))

    def __call__(self, psi):
        out = torch.empty(psi.shape, dtype=torch.complex128, device="cuda")
        N1, N2, N3 = self.b.Ns
        step = max(1, int(4e8 // (16 * self.b.Npoints)))
        for j in range(0, psi.shape[0], step):
            x = psi[j:j + step].to(torch.complex128)
            f = torch.fft.fftn(self.grid(x) * self.V.view(N3, N2, N1), dim=(1, 2, 3))
            out[j:j + step] = f.reshape(x.shape[0], -1)[:, self.idx] + 0.5 * self.gk2 * x
        x = psi.to(torch.complex128)
        for a in range(0, self.pos.shape[1], 8):
            ph = torch.exp(-1j * (self.g @ self.pos[:, a:a + 8])).T                       # (8, Ngw)
            beta = (ph[:, None, :] * self.radial[None]).reshape(-1, ph.shape[1])          # (8 * 5, Ngw)
            c = (beta.conj() @ x.T).view(ph.shape[0], 5, -1)
            c = torch.einsum("ij,ajb->aib", self.D, c).reshape(-1, x.shape[0])
            out += c.T @ beta
        return out

    def density(self, psi, w):
        rho = torch.zeros(self.b.Npoints, dtype=torch.float64, device="cuda")
        step = max(1, int(4e8 // (16 * self.b.Npoints)))
        for j in range(0, psi.shape[0], step):
            f = self.grid(psi[j:j + step].to(torch.complex128)).reshape(-1, self.b.Npoints) * self.b.Npoints
            rho += (torch.from_numpy(w[j:j + step]).cuda()[:, None] * (f.real ** 2 + f.imag ** 2)).sum(dim=0)
        return rho / self.b.CellVolume


def _lowest(T, G, k):
    """The k lowest pairs of T s = lam G s, s' G s = 1 (Hermitian, upper triangles)."""
    T = torch.triu(T) + torch.triu(T, 1).conj().T
    G = torch.triu(G) + torch.triu(G, 1).conj().T
    L = torch.linalg.cholesky(G)
    Li = torch.linalg.solve_triangular(L, torch.eye(len(T), dtype=T.dtype, device=T.device), upper=False)
    lam, Z = torch.linalg.eigh(Li @ T @ Li.conj().T)
    return lam[:k], Li.conj().T @ Z[:, :k]


def _lobpcg(op, X, iters):
    """LOBPCG with Q = [X W P], the steps of diag_LOBPCG.jl:51-225 (rows are bands)."""
    nb = X.shape[0]

    def inner(A, B):
        return A.conj() @ B.T

    def orth(A, HA):
        R = torch.linalg.cholesky(inner(A, A)).conj().T
        Ri = torch.linalg.solve_triangular(R, torch.eye(nb, dtype=R.dtype, device=R.device), upper=True)
        return Ri.T @ A, Ri.T @ HA
    HX = op(X)
    P = HP = None
    for it in range(iters):
        W = (HX - inner(X, HX).T @ X) / (1.0 + op.gk2)
        W, HW = orth(W, op(W))
        Q = torch.cat([X, W] + ([P] if it else []))
        HQ = torch.cat([HX, HW] + ([HP] if it else []))
        _, U = _lowest(inner(Q, HQ), inner(Q, Q), nb)
        X, HX = U.T @ Q, U.T @ HQ
        P, HP = orth(U[nb:].T @ Q[nb:], U[nb:].T @ HQ[nb:]) if it else (W, HW)
    S = inner(X, HX)
    lam, V = torch.linalg.eigh(0.5 * (S + S.conj().T))
    return lam, V.T @ X


def exact(case, seed):
    kind = case["kind"]
    if kind == "rr":
        Q, HQ, U = _rr_inputs(case, seed)
        Qd = Q.to(torch.complex128)
        return {"T": (Qd.conj() @ HQ.to(torch.complex128).T).T.contiguous(), "G": (Qd.conj() @ Qd.T).T.contiguous(),
                "X": U @ Qd}
    if kind == "eigh":
        T, G = _eigh_inputs(case, seed)
        lam, S = _lowest(T.T.contiguous(), G.T.contiguous(), case["k"])     # run() hands the column-major matrices over
        return {"lam": lam, "P": S @ S.conj().T}
    if kind == "multik":
        b, gk, _ = _basis(*_of(case))
        op, pos, outs = _Op(case, seed), _positions(case, seed), []
        for ik in range(b.Nkpt):
            op.set_k(ik, AL, pos, gk[ik])
            outs.append(op(_block(case["bands"], b.Gk2[ik], seed, 10 + ik, case["dtype"])).reshape(-1))
        return torch.cat(outs)
    op = _Op(case, seed)
    psi = _block(case["bands"], op.b.Gk2[0], seed, 1, "fp64" if kind == "host" else case["dtype"])
    if kind == "opH":
        return op(psi)
    if kind == "host":
        return op(psi).cpu().numpy().T
    if kind == "rhoe":
        return op.density(psi, _weights(case["bands"]))
    lam, X = _lobpcg(op, psi.to(torch.complex128), case["iters"])
    return {"evals": lam.cpu().numpy(), "rho": op.density(X, _weights(case["bands"]))}


def tolerance(case):
    """About four times what the path differs by from the 64-bit results
    (measured: op_H and the density 9e-7 in 32 bits, 8e-16 in 64; the
    products 4.5e-6 and 6e-15; the eigenproblem 3e-14), with room for the
    larger shapes; whole solves pass rounding on from step to step."""
    kind, mixed = case["kind"], case.get("dtype") == "mixed"
    if kind == "eigh":
        return {"rel": 1e-12, "max": 1e-10}
    if kind == "lobpcg":
        return {"rel": 2e-5, "max": 1e-3} if mixed else {"rel": 1e-10, "max": 1e-8}
    if kind == "rr":
        return {"rel": 2e-5, "max": 1e-3} if mixed else {"rel": 3e-14, "max": 1e-12}
    return {"rel": 3e-6, "max": 1e-4} if mixed else {"rel": 1e-14, "max": 1e-12}
