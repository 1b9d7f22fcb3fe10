"""Performance cases of the MDFT engine: what its users run, over the range of sizes they run.

A Fortran or Python host evaluates the functional and its gradient on its grid (FP64, or the
mixed form with FP32 vectors on its side), minimises, or hands a solute over to be solved;
the warm-start network is trained with its own forward and backward pass.  Grids are the
engine's 2^a 3^b lengths at the 0.5 A spacing of the uneven batch (0.625 A for the single
ion, 0.375 A at mmax 5), solutes the seeded random walks of the benchmark, the solvent the
synthetic water with its seeded c(k).

`exact` restates the functional (without the reference's single-precision flushes) and the
network in torch float64.
"""
from __future__ import annotations

import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "mdft-dev_general_b200"))

from mdft_b200 import engine as E  # noqa: E402
from mdft_b200 import synth  # noqa: E402
from mdft_b200 import warmstart as W  # noqa: E402

DEV = "cuda"
SOLVENT = synth.Solvent()
CK_SEED = 20260001
HISTORY = 5  # L-BFGS pairs, the benchmark's m


def listed():
    return [
        # the smallest system of the tests: one LJ-ion-sized box, all latency and launches
        dict(name="fp64_16_m1", kind="eval", prec="fp64", nx=16, ny=16, nz=16, mmax=1, dx=0.5, nsite=1),
        # the single ion at the centre of a 20 A box, the reference's own CPU-sized system
        dict(name="fp64_32_m1", kind="eval", prec="fp64", nx=32, ny=32, nz=32, mmax=1, dx=0.625, nsite=1),
        # an elongated box through host arrays, as the Fortran host calls energy_and_gradient
        dict(name="fp64_host_24x36x48_m2", kind="host", prec="fp64", nx=24, ny=36, nz=48, mmax=2, dx=0.5, nsite=6),
        # the workload of the benchmark: a 24-site molecule, plain FP64
        dict(name="fp64_64_m3", kind="eval", prec="fp64", nx=64, ny=64, nz=64, mmax=3, dx=0.5, nsite=24),
        # the largest grid of the uneven batch, low angular order
        dict(name="fp64_96_m1", kind="eval", prec="fp64", nx=96, ny=96, nz=96, mmax=1, dx=0.5, nsite=40),
        # the highest angular order, FP64, small box
        dict(name="fp64_32_m5", kind="eval", prec="fp64", nx=32, ny=32, nz=32, mmax=5, dx=0.375, nsite=12),
        # mixed precision, the benchmark's grid
        dict(name="mixed_64_m3", kind="eval", prec="mixed", nx=64, ny=64, nz=64, mmax=3, dx=0.5, nsite=24),
        # mixed precision at the packed cluster's angular order and spacing
        dict(name="mixed_64_m5", kind="eval", prec="mixed", nx=64, ny=64, nz=64, mmax=5, dx=0.375, nsite=59),
        # L-BFGS steps from a density at hand (a restart), plain FP64
        dict(name="lbfgs_fp64_48_m3", kind="minimize", prec="fp64", nx=48, ny=48, nz=48, mmax=3, dx=0.5, nsite=12, iters=6),
        # the same with the benchmark's grid and default form: FP32 vectors, BF16 history
        dict(name="lbfgs_mixed_64_m3", kind="minimize", prec="mixed", nx=64, ny=64, nz=64, mmax=3, dx=0.5, nsite=24, iters=16),
        # a solute in, its free energy out: external potential, guess, a fixed number of L-BFGS
        # iterations (as the reference's benchmark minimizer), pressure correction
        dict(name="solve_fp64_48_m3", kind="solve", prec="fp64", nx=48, ny=48, nz=48, mmax=3, dx=0.5, nsite=24, iters=12),
        # forward and backward of the warm-start network on its training grid
        dict(name="warm_gradients_48", kind="warm", prec="fp32", nx=48, ny=48, nz=48, mmax=3, dx=0.5, nsite=20),
    ]


LENGTHS = (8, 12, 16, 18, 24, 32, 36, 48, 54, 64, 72, 96)
MOST_VALUES = 64 ** 3 * 84  # orientations x points of a drawn system: the benchmark's


def _sizes(mmax):
    no = (mmax + 1) * (2 * mmax + 1) * (2 * (mmax // 2) + 1)
    np_ = sum((2 * m + 1) * (m // 2 + 1) for m in range(mmax + 1))
    return no, np_


def draw(rng):
    kind = rng.choice(("eval", "eval", "eval", "eval", "host", "minimize", "solve", "warm"))
    if kind == "warm":
        n = rng.choice((16, 24, 32, 40, 48))
        return dict(kind="warm", prec="fp32", nx=n, ny=n, nz=n, mmax=3, dx=0.5, nsite=rng.randint(1, 30))
    while True:
        mmax = rng.choice((0, 1, 1, 2, 3, 3, 4, 5))
        if kind == "solve":
            mmax = rng.choice((1, 3))
        nx = rng.choice(LENGTHS)
        dims = [nx, nx, nx]
        if kind != "solve" and rng.random() < 0.4:  # boxes that are not cubes
            dims = [rng.choice([v for v in LENGTHS if nx / 2 <= v <= 2 * nx]) for _ in range(3)]
        no, _ = _sizes(mmax)
        total = dims[0] * dims[1] * dims[2]
        if kind == "solve" and nx not in (24, 32, 48):
            continue
        if kind == "minimize" and mmax > 3:
            continue
        if total * no <= MOST_VALUES // (3 if kind in ("host", "minimize") else 1):
            break
    c = dict(kind=kind, prec=rng.choice(("fp64", "mixed")) if kind in ("eval", "minimize") else "fp64",
             nx=dims[0], ny=dims[1], nz=dims[2], mmax=mmax, dx=0.375 if mmax > 3 else 0.5, nsite=rng.randint(1, 40))
    if kind == "minimize":
        c["iters"] = rng.randint(2, 6)
    if kind == "solve":
        c["iters"] = rng.randint(4, 12)
    return c


# ----------------------------------------------------------------------------
# inputs
_CK = {}


def _ck_params(case):
    if case["mmax"] > 3:
        return case["mmax"], 15.0, 0.05
    return case["mmax"], 12.0, 0.02


def _ck_file(case):
    """The c(k) file of the solvent at this angular order (one per process)."""
    key = _ck_params(case)
    if key not in _CK:
        d = tempfile.mkdtemp(prefix="mdft_ck_")
        mmax, kmax, dk = key
        _CK[key] = synth.make_ck_file(os.path.join(d, "ck.txt"), mmax, seed=CK_SEED, kmax=kmax, dk=dk)
    return _CK[key]


def _box(case):
    return tuple(case["dx"] * case[k] for k in ("nx", "ny", "nz"))


def _rvdw(case):
    return min(10.0, 0.49 * min(_box(case)))


def _solute(case, seed):
    if case["nsite"] == 1:
        s = synth.ion_solute()
    else:
        s = synth.random_walk_solute(case["nsite"], seed=1000 + seed, radius=min(6.0, max(2.5, 0.25 * min(_box(case)))),
                                     min_sep=0.9)
    s.xyz = synth.center_solute(s.xyz, _box(case))
    return s


def _orientations(mmax):
    """cos/sin of the quadrature angles per orientation, theta slowest, psi fastest."""
    x, _ = np.polynomial.legendre.leggauss(mmax + 1)
    theta = np.arccos(x[::-1])
    phi = np.arange(2 * mmax + 1) * 2 * math.pi / (2 * mmax + 1)
    npsi = 2 * (mmax // 2) + 1
    psi = np.arange(npsi) * math.pi / npsi
    t, p, s = np.meshgrid(theta, phi, psi, indexing="ij")
    return t.reshape(-1), p.reshape(-1), s.reshape(-1)


def _fields(case, seed):
    """External potential and density amplitude [nz, ny, nx, no] around the seeded solute:
    Lennard-Jones repulsion and attraction, a field on the molecular axis, and xi near
    exp(-v / 2 kT) with the noise of an unconverged density."""
    sol = _solute(case, seed)
    no, _ = _sizes(case["mmax"])
    lx, ly, lz = _box(case)
    dev = torch.device(DEV)
    ax = [torch.arange(case[k], dtype=torch.float64, device=dev) * case["dx"] for k in ("nx", "ny", "nz")]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    lj = torch.zeros_like(x)
    field = torch.zeros((3,) + tuple(x.shape), dtype=torch.float64, device=dev)
    for k in range(len(sol.q)):
        d = [a - float(p) for a, p in zip((x, y, z), sol.xyz[k])]
        d = [v - L * torch.round(v / L) for v, L in zip(d, (lx, ly, lz))]
        r2 = (d[0] ** 2 + d[1] ** 2 + d[2] ** 2).clamp(min=0.25)
        s6 = (0.5 * (float(sol.sig[k]) + SOLVENT.sig[0])) ** 6 / r2 ** 3
        lj += 4.0 * math.sqrt(float(sol.eps[k]) * SOLVENT.eps[0]) * s6 * (s6 - 1.0)
        w = float(sol.q[k]) * 40.0 / (r2 + 4.0) ** 1.5
        for j in range(3):
            field[j] += w * d[j]
    t, p, _ = _orientations(case["mmax"])
    if no == 1:
        t, p = np.zeros(1), np.zeros(1)
    u = [torch.tensor(v, device=dev) for v in (np.sin(t) * np.cos(p), np.sin(t) * np.sin(p), np.cos(t))]
    v = lj[..., None] + sum(field[j][..., None] * u[j] for j in range(3))
    v = v.clamp(max=694.0)
    g = torch.Generator(device=dev)
    g.manual_seed(77000 + seed)
    xi = torch.exp((v * (-0.5 / SOLVENT.kT)).clamp(min=-40.0, max=0.7))
    xi = xi * (1.0 + 0.1 * torch.randn(v.shape, dtype=torch.float64, device=dev, generator=g))
    return v.contiguous(), xi.contiguous()


def _engine(case, seed):
    return E.Engine((case["nx"], case["ny"], case["nz"]), _box(case), case["mmax"], _ck_file(case),
                    temperature=SOLVENT.temperature, n0=SOLVENT.n0,
                    precision=E.PREC_MIXED if case["prec"] == "mixed" else E.PREC_FP64)


def _warm_inputs(case, seed):
    """Input channels, target and mask as the training set holds them: compressed Lennard-Jones
    and electrostatic potentials, the site density, a smooth log-density around the solute."""
    sol = _solute(case, seed)
    dev = torch.device(DEV)
    lx = _box(case)[0]
    a = torch.arange(case["nx"], dtype=torch.float32, device=dev) * case["dx"]
    z, y, x = torch.meshgrid(a, a, a, indexing="ij")
    lj, q, rho = (torch.zeros_like(x) for _ in range(3))
    for k in range(len(sol.q)):
        d = [v - float(p) for v, p in zip((x, y, z), sol.xyz[k])]
        r2 = sum((v - lx * torch.round(v / lx)) ** 2 for v in d).clamp(min=0.25)
        s6 = (0.5 * (float(sol.sig[k]) + SOLVENT.sig[0])) ** 6 / r2 ** 3
        lj += 4.0 * math.sqrt(float(sol.eps[k]) * SOLVENT.eps[0]) * s6 * (s6 - 1.0)
        q += 1389.35 * float(sol.q[k]) / torch.sqrt(r2 + 0.5)
        rho += torch.exp(-2.0 * r2)
    kT = SOLVENT.kT
    feat = torch.stack([torch.asinh((lj / kT).clamp(max=1e4)) / 4, torch.asinh(q / kT) / 4, rho]).contiguous()
    g = torch.Generator(device=dev)
    g.manual_seed(99000 + seed)
    tgt = torch.stack([(-lj / kT).clamp(min=-8.0, max=1.0)] + [0.3 * torch.tanh(q / kT)] * 3)
    tgt = (tgt + 0.05 * torch.randn(tgt.shape, device=dev, generator=g)).contiguous()
    mask = (lj < 30.0 * kT).to(torch.float32).contiguous()
    return feat, tgt, mask


def prepare(case, seed):
    if case["kind"] == "warm":
        feat, tgt, mask = _warm_inputs(case, seed)
        params, _ = W.load_params()
        return dict(kind="warm", net=W.WarmNet(case["nx"], params=params), feat=feat, tgt=tgt, mask=mask)
    eng = _engine(case, seed)
    if case["kind"] == "solve":
        return dict(kind="solve", eng=eng, sol=_solute(case, seed), rvdw=_rvdw(case), iters=case["iters"])
    v, xi = _fields(case, seed)
    eng.set_vext(v.cpu().numpy())
    st = dict(kind=case["kind"], eng=eng)
    if case["kind"] == "host":
        st.update(xi=xi.cpu().numpy(), df=np.empty(tuple(xi.shape)))
    elif case["kind"] == "minimize":
        st.update(start=xi, xi=torch.empty_like(xi), iters=case["iters"])
        if case["prec"] == "mixed":
            st["xi16"] = torch.empty(xi.shape, dtype=torch.bfloat16, device=DEV)
    else:
        st.update(xi=xi, df=torch.empty_like(xi))
        if case["prec"] == "mixed":
            st["df32"] = torch.empty(xi.shape, dtype=torch.float32, device=DEV)
    torch.cuda.synchronize()
    return st


def run(st):
    if st["kind"] == "warm":
        g, loss = st["net"].gradients(st["feat"].data_ptr(), st["tgt"].data_ptr(), st["mask"].data_ptr())
        return dict(gradients=g, loss=loss)
    eng = st["eng"]
    if st["kind"] == "solve":
        r = eng.solve(st["sol"], SOLVENT, rvdw=st["rvdw"], m=HISTORY, pgtol=1e-9, ftol_abs=-1.0, itermax=st["iters"])
        return {k: float(r[k]) for k in ("dG", "f", "pmv", "lj_tail", "deltaN")}
    if st["kind"] == "host":
        f, df, terms = eng.energy_and_gradient(st["xi"], df_out=st["df"])
        return dict(f=f, df=df, terms=terms)
    if st["kind"] == "minimize":
        st["xi"].copy_(st["start"])
        torch.cuda.current_stream().synchronize()  # the engine has a stream of its own
        r = eng.minimize_device(st["xi"].data_ptr(), m=HISTORY, pgtol=1e-12, ftol_abs=-1.0, itermax=st["iters"],
                                precision=E.PREC_MIXED if "xi16" in st else E.PREC_FP64, polish=0)
        if "xi16" in st:
            # single values of an unconverged FP32 path are good to 1e-3 (its history is BF16)
            st["xi16"].copy_(st["xi"])
            return dict(f=r["f"], xi=st["xi16"])
        return dict(f=r["f"], xi=st["xi"])
    f, terms = eng.energy_and_gradient_device(st["xi"].data_ptr(), st["df"].data_ptr())
    if "df32" in st:  # the host's FP32 vectors, as a mixed minimiser keeps them
        st["df32"].copy_(st["df"])
        return dict(f=f, df=st["df32"], terms=[float(t) for t in terms])
    return dict(f=f, df=st["df"], terms=terms)


def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "warm":
        s = case["nx"] ** 3
        fwd = 0
        for k, _, _, ci, co, _, _ in _layers():
            taps, vox = {0: (27, 1), 1: (8, 1), 2: (1, 1), 3: (1, 1)}[k]
            lvl = {(3, 16): 0, (16, 16): 0, (16, 32): 1, (32, 32): 1, (32, 64): 2, (64, 64): 2, (64, 128): 3, (128, 128): 3,
                   (128, 64): 2, (64, 32): 1, (32, 16): 0, (16, 4): 0}[(ci, co)]
            fwd += 2 * taps * ci * co * (s // 8 ** lvl)
        return dict(bytes=4 * s * (3 + 4 + 1) + 4 * 906772, flops=3 * fwd)
    no, np_ = _sizes(case["mmax"])
    ang = 2 * (2 * n * no * 2 * np_)
    fft = 2 * np_ * 5 * n * math.log2(n)
    M = case["mmax"]
    rot = sum((2 * m + 1) ** 2 * (m // 2 + 1) for m in range(M + 1))
    ncoef = sum((2 * (k // 2) + 1) for m in range(M + 1) for chi in range(-m, m + 1) for _ in range(m // 2 + 1)
                for k in range(abs(chi), M + 1))
    flops = ang + fft + n * (2 * rot * 4 + ncoef * 8)
    field = 8 * n * no
    if case["kind"] in ("eval", "host"):
        return dict(bytes=3 * field + (field // 2 if case["prec"] == "mixed" else 0), flops=flops)
    # per iteration: the evaluation's four fields and the history pairs, at the vectors' widths
    it = case["iters"]
    vec, hist = (field // 2, field // 4) if case["prec"] == "mixed" else (field, field)
    return dict(bytes=(it + 1) * 4 * vec + it * 2 * HISTORY * hist, flops=(it + 1) * flops)


# ----------------------------------------------------------------------------
# the functional in torch float64
def _wigner(m, a, b, th):
    """d^m_{ab}(theta), Wigner's sum."""
    out = np.zeros_like(th)
    f = math.factorial
    c, s = np.cos(th / 2), np.sin(th / 2)
    for k in range(max(0, a - b), min(m + a, m - b) + 1):
        out += (-1) ** k / (f(m + a - k) * f(m - b - k) * f(k) * f(k - a + b)) * c ** (2 * m + a - b - 2 * k) * s ** (2 * k - a + b)
    return math.sqrt(f(m + a) * f(m - a) * f(m + b) * f(m - b)) * out


def _rotations(q, M):
    """R[l][m + l][m1 + l] of the frame of each q (3, n), by the recursion of the reference's
    module_rotation (src/module_rotation.f90:119-247) in complex128."""
    n = q.shape[1]
    zero = (q == 0).all(0)
    r3 = torch.where(zero, torch.tensor([[0.0], [0.0], [1.0]], dtype=q.dtype, device=q.device), q)
    inplane = (r3[0] != 0) | (r3[1] != 0)
    z = torch.zeros(n, dtype=q.dtype, device=q.device)
    r2 = torch.where(inplane, torch.stack([-r3[1], r3[0], z]), torch.stack([z, r3[2], -r3[1]]))
    r3 = r3 / r3.norm(dim=0)
    r2 = r2 / r2.norm(dim=0)
    r1 = torch.linalg.cross(r2, r3, dim=0)
    c = torch.complex
    h = math.sqrt(0.5)
    R = [[[torch.ones(n, dtype=torch.complex128, device=q.device)]]]
    if M >= 1:
        R.append([[c((r2[1] + r1[0]) / 2, (r1[1] - r2[0]) / 2), c(r3[0] * h, r3[1] * h), c((r2[1] - r1[0]) / 2, (-r1[1] - r2[0]) / 2)],
                  [c(r1[2] * h, -r2[2] * h), c(r3[2], z), c(-r1[2] * h, -r2[2] * h)],
                  [c((r2[1] - r1[0]) / 2, (r1[1] + r2[0]) / 2), c(-r3[0] * h, r3[1] * h), c((r2[1] + r1[0]) / 2, (r2[0] - r1[1]) / 2)]])
    for l in range(2, M + 1):
        U = lambda m, m1: R[l - 1][m + l - 1][m1 + l - 1] if abs(m) < l and abs(m1) < l else None  # noqa: E731
        X = lambda m, m1: R[1][m + 1][m1 + 1]  # noqa: E731
        T = [[None] * (2 * l + 1) for _ in range(2 * l + 1)]
        for m in range(-l, l + 1):
            for m1 in range(1 if m > 0 else 0, l + 1):
                if m1 < l:
                    den, x1 = math.sqrt((l + m1) * (l - m1)), 0
                    a = math.sqrt((l + m) * (l - m)) / den
                    b = lambda k: math.sqrt((l + k) * (l + k - 1)) / (math.sqrt(2.0) * den)  # noqa: E731
                    u1 = m1
                else:
                    den, x1 = math.sqrt(2 * l * (2 * l - 1)), 1
                    a = math.sqrt(2.0) * math.sqrt((l + m) * (l - m)) / den
                    b = lambda k: math.sqrt((l + k) * (l + k - 1)) / den  # noqa: E731
                    u1 = m1 - 1
                v = 0
                for cf, xm, um in ((a, 0, m), (b(m) if l + m >= 1 else 0.0, 1, m - 1), (b(-m) if l - m >= 1 else 0.0, -1, m + 1)):
                    u = U(um, u1)
                    if u is not None and cf != 0.0:
                        v = v + cf * X(xm, x1) * u
                T[m + l][m1 + l] = v
                if m == 0 and m1 == 0:
                    T[l][l] = v.conj()
                else:
                    T[-m + l][-m1 + l] = (-1) ** (m + m1) * v.conj()
        R.append(T)
    return R


def _excess(case, xi, ck):
    """(sum for F_exc's integrand, gradient) of the excess term at xi [nz, ny, nx, no]."""
    M = case["mmax"]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    N = nx * ny * nz
    no, np_ = _sizes(M)
    dev = xi.device
    t, p, s = _orientations(M)
    _, wt = np.polynomial.legendre.leggauss(M + 1)
    nphi, npsi = 2 * M + 1, 2 * (M // 2) + 1
    wt = np.repeat(wt[::-1] / 2, nphi * npsi)
    proj = [(m, mup, mu) for m in range(M + 1) for mup in range(-m, m + 1) for mu in range(0, m + 1, 2)]
    index = {v: i for i, v in enumerate(proj)}
    A = np.empty((no, np_), dtype=complex)
    B = np.empty((np_, no), dtype=complex)
    for i, (m, mup, mu) in enumerate(proj):
        d = math.sqrt(2 * m + 1) * _wigner(m, mup, mu, t)
        ph = np.exp(1j * (mup * p + mu * s))
        A[:, i] = d * wt / (nphi * npsi) * ph
        B[i] = (1 if mu == 0 else 2) * d * np.conj(ph)
    A, B = torch.tensor(A, device=dev), torch.tensor(B, device=dev)
    rho0 = SOLVENT.rho0
    drho = rho0 * (xi * xi - 1.0)
    pl = (drho.reshape(N, no).to(torch.complex128) @ A).T.reshape(np_, nz, ny, nx)
    del drho
    pl = torch.fft.ifftn(pl, dim=(1, 2, 3), norm="forward").reshape(np_, N)
    kz, ky, kx = torch.meshgrid(*[torch.arange(n, device=dev) for n in (nz // 2 + 1, ny, nx)], indexing="ij")
    kx, ky, kz = kx.reshape(-1), ky.reshape(-1), kz.reshape(-1)
    mx, my, mz = (-kx) % nx, (-ky) % ny, (-kz) % nz
    # the q of each pair: the member met first in the planes that hold both
    keep = ~(((kz == 0) | (2 * kz == nz)) & (ky * nx + kx > my * nx + mx))
    kx, ky, kz, mx, my, mz = (v[keep] for v in (kx, ky, kz, mx, my, mz))
    iq, im = (kz * ny + ky) * nx + kx, (mz * ny + my) * nx + mx
    nyq = (2 * kx == nx) | (2 * ky == ny) | (2 * kz == nz)
    lx, ly, lz = _box(case)
    sg = lambda k, n, L: torch.where(k <= n // 2, k, k - n).to(torch.float64) * (2 * math.pi / L)  # noqa: E731
    q = torch.stack([sg(kx, nx, lx), sg(ky, ny, ly), sg(kz, nz, lz)])
    R = _rotations(q, M)
    dq, dm = pl[:, iq], pl[:, im]
    rq, rm = torch.empty_like(dq), torch.empty_like(dm)
    for (m, chi, mu), i in index.items():
        rq[i] = sum(dq[index[(m, k, mu)]] * R[m][k + m][chi + m] for k in range(-m, m + 1))
        rm[i] = (-1) ** m * sum(dm[index[(m, k, mu)]] * R[m][k + m][-chi + m] for k in range(-m, m + 1))
    qs, tuples, vals = ck
    col = {tp: i for i, tp in enumerate(tuples)}
    vals = torch.tensor(vals, device=dev)
    eff = q.norm(dim=0) / (qs[3] - qs[2])
    lo = eff.floor().to(torch.int64)
    al = (eff - lo).to(torch.complex128)
    gq, gm = torch.zeros_like(dq), torch.zeros_like(dm)
    for (m, chi, mu), i in index.items():
        for n in range(abs(chi), M + 1):
            for nu in range(-(n // 2) * 2, n + 1, 2):
                cv = vals[:, col[(m, n, mu, nu, chi)]].conj() * ((-1) ** (chi + nu) if nu < 0 else (-1) ** n)
                c = (1 - al) * cv[lo] + al * cv[lo + 1]
                j = index[(n, chi, abs(nu))]
                if nu < 0:
                    gq[i] += c * rq[j]
                    gm[i] += c * rm[j]
                else:
                    gq[i] += c * rm[j].conj()
                    gm[i] += c * rq[j].conj()
    del rq, rm, dq, dm
    self_ = iq == im
    for (m, mup, mu), i in index.items():
        a = sum(gq[index[(m, k, mu)]] * R[m][mup + m][k + m].conj() for k in range(-m, m + 1))
        b = (-1) ** m * sum(gm[index[(m, k, mu)]] * R[m][mup + m][-k + m].conj() for k in range(-m, m + 1))
        b = torch.where(self_ & nyq, b.conj(), b)
        pl[i, iq] = a
        pl[i, im] = b  # self-conjugate points keep the -q result
    del gq, gm, R
    pl = torch.fft.fftn(pl.reshape(np_, nz, ny, nx), dim=(1, 2, 3)).reshape(np_, N) / N
    w = torch.tensor(wt / nphi / (npsi * 2) * 8 * math.pi ** 2, device=dev)
    v = (pl.T.real @ B.real - pl.T.imag @ B.imag).reshape(nz, ny, nx, no)
    v = v * w * (-SOLVENT.kT * 2 * 4 * math.pi ** 2 / 2 / SOLVENT.n0)
    return ((xi * xi * rho0 - rho0) * v).sum(), 2 * rho0 * xi * v, w


def _functional(case, v, xi, ck):
    kT, rho0 = SOLVENT.kT, SOLVENT.rho0
    dv = case["dx"] ** 3
    sexc, df, w = _excess(case, xi, ck)
    x2 = xi * xi
    occ = x2 * rho0 > 2.220446049250313e-16
    lg = torch.log(torch.where(occ, x2, torch.ones_like(x2)))
    fid = kT * dv * (w * torch.where(occ, rho0 * (x2 * lg - x2 + 1.0), torch.full_like(x2, rho0))).sum()
    fext = dv * (w * torch.where(occ, rho0 * x2 * v, torch.zeros_like(x2))).sum()
    fexc = 0.5 * dv * sexc
    df += torch.where(occ, 2 * w * rho0 * xi * (kT * lg + v), torch.zeros_like(x2))
    terms = [float(fid), float(fext), float(fexc), 0.0]
    return sum(terms), df, terms


_TABLE = {}


def _table(case):
    key = _ck_params(case)
    if key not in _TABLE:
        q, tuples, vals = synth.synthetic_ck(key[0], seed=CK_SEED, kmax=key[1], dk=key[2])
        _TABLE[key] = (q, tuples, vals)
    return _TABLE[key]


def _layers():
    conv, down, up, head = 0, 1, 2, 3
    return [(conv, 0, 1, 3, 16, -1, 1), (conv, 1, 2, 16, 16, -1, 1), (down, 2, 3, 16, 32, -1, 1), (conv, 3, 4, 32, 32, -1, 1),
            (down, 4, 5, 32, 64, -1, 1), (conv, 5, 6, 64, 64, -1, 1), (down, 6, 7, 64, 128, -1, 1), (conv, 7, 8, 128, 128, -1, 1),
            (up, 8, 9, 128, 64, 6, 0), (conv, 9, 10, 64, 64, -1, 1), (up, 10, 11, 64, 32, 4, 0), (conv, 11, 12, 32, 32, -1, 1),
            (up, 12, 13, 32, 16, 2, 0), (conv, 13, 14, 16, 16, -1, 1), (head, 14, 15, 16, 4, -1, 0)]


def _warm_exact(case, seed):
    feat, tgt, mask = (v.double() for v in _warm_inputs(case, seed))
    p, _ = W.load_params()  # BF16 weights; biases as shipped
    flat = torch.tensor(p.astype(np.float64), device=DEV, requires_grad=True)
    F = torch.nn.functional
    x, off = {0: feat[None]}, 0
    for k, xi, yi, ci, co, skip, gelu in _layers():
        shape = ((co, ci) if k != 2 else (ci, co)) + ((3,) * 3 if k == 0 else (1,) * 3 if k == 3 else (2,) * 3)
        n = int(np.prod(shape))
        w, b = flat[off:off + n].reshape(shape), flat[off + n:off + n + co]
        off += n + co
        a = x[xi]
        if k == 0:
            y = F.conv3d(F.pad(a, (1,) * 6, mode="circular"), w, b)
        elif k == 1:
            y = F.conv3d(a, w, b, stride=2)
        elif k == 2:
            y = F.conv_transpose3d(a, w, b, stride=2) + x[skip]
        else:
            y = F.conv3d(a, w, b)
        x[yi] = F.gelu(y) if gelu else y
    loss = (((x[15][0] - tgt) ** 2).sum(0) * mask).sum() / (4.0 * case["nx"] ** 3)
    loss.backward()
    return dict(gradients=flat.grad, loss=float(loss))


def exact(case, seed):
    if case["kind"] == "warm":
        return _warm_exact(case, seed)
    if case["kind"] in ("minimize", "solve"):
        return None  # iterates of a minimisation, not values of a formula
    v, xi = _fields(case, seed)
    f, df, terms = _functional(case, v, xi, _table(case))
    return dict(f=f, df=df, terms=terms if case["prec"] == "mixed" else np.array(terms))
