"""Performance cases of the solver: what a program does with it, through the
Python binding's entry points, over the range of grids it is used on.

listed() names fixed cases, draw() gives further ones of the same ranges;
prepare() builds what a program holds before the call (medium, sources, the
solver of that grid), run() is one pass and work() the bytes and operations
it cannot do without.  exact() computes a pass's outputs in 64 bits with
plain torch.

Kinds of case:
  op         the 7-point operator (or its adjoint) on one vector
  prec       the preconditioner (or its adjoint) on one complex128 vector
  prec_batch the complex64 preconditioner on a batch, its output kept in
             complex64 as flexible GMRES keeps its Z basis
  solve      solves with a factored medium
  step       a new medium, its factor and the solves, as one inversion or
             survey step does
  group      new media and one grouped solve of uneven grids
  gradient   misfit and gradient: batched forward and adjoint solves
  reference  the reference's own formulation (K = I - dL L0^{-1}, complex128)
             by FGMRES
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "iterative-helmholtz-solver-with-pardiso_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import helm3d  # noqa: E402
from helm3d import media  # noqa: E402

# preconditioner shifts in use: the FFT z-transform needs damping, the PML
# eigenbasis is exact along z
BETA = {"fft": 0.25, "eigen": 0.01}
C_REF = 1280.0      # m/s, the reference's homogeneous sound speed
HZ_REF = 4.0        # Hz, its frequency
LEN_REF = 3200.0    # m, its domain


def listed():
    return [
        # the smallest call: one operator application on a test-sized grid
        dict(name="op_20", kind="op", nx=20, ny=20, nz=20, pml=4, adjoint=False),
        # one adjoint operator application on the largest grid
        dict(name="op_adjoint_200", kind="op", nx=200, ny=200, nz=200, pml=16, adjoint=True),
        # the reference's preconditioner (z-FFT, complex128) at the 64^3 configuration
        dict(name="prec_fft_64", kind="prec", nx=64, ny=64, nz=64, pml=8, zt="fft", adjoint=False),
        # the adjoint preconditioner of an odd, uneven grid, eigenbasis
        dict(name="prec_adjoint_uneven", kind="prec", nx=57, ny=48, nz=53, pml=8, zt="eigen", adjoint=True),
        # the complex64 preconditioner on a full batch inside a caller's own iteration
        dict(name="prec_batch_96", kind="prec_batch", nx=96, ny=96, nz=96, pml=8, zt="fft", nrhs=16),
        # a single small solve, where launches and latency count
        dict(name="solve_20", kind="solve", nx=20, ny=20, nz=20, pml=4, prec="c64", zt="eigen", nrhs=1,
             medium="layered", restart=20, tol=1e-9),
        # the homogeneous 64^3 configuration, plain complex128 FFT-z path
        dict(name="solve_64_fft_c128", kind="solve", nx=64, ny=64, nz=64, pml=8, prec="c128", zt="fft", nrhs=1,
             medium="homogeneous", restart=20, tol=1e-8),
        # the heterogeneous 128^3 step: set-up, factor and 16 batched sources
        dict(name="step_128", kind="step", nx=128, ny=128, nz=128, pml=12, prec="c64", zt="eigen", nrhs=16,
             medium="layered", restart=20, tol=1e-8),
        # the headline 200^3 medium, its factor and 4 sources
        dict(name="step_200", kind="step", nx=200, ny=200, nz=200, pml=16, prec="c64", zt="eigen", nrhs=4,
             medium="layered", restart=20, tol=1e-8),
        # uneven grids, each with its own medium and source, as one group
        dict(name="group_uneven", kind="group", nx=112, ny=96, nz=64, pml=8, grids=4, nrhs=1, restart=20, tol=1e-8),
        # misfit and gradient of 8 sources and a plane of receivers
        dict(name="gradient_96", kind="gradient", nx=96, ny=96, nz=96, pml=8, nrhs=8, nrecv=24, restart=30,
             tol=1e-10),
        # the reference's formulation on the reference's 58^3 grid
        dict(name="reference_58", kind="reference", nx=58, ny=58, nz=58, pml=4, spg=4, restart=30,
             tol=1e-10),
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    return dict(nx=_side(rng, lo, hi), ny=_side(rng, lo, hi), nz=_side(rng, lo, hi))


def draw(rng):
    kind = rng.choice(["op", "prec", "prec_batch", "solve", "step", "step", "group", "gradient", "reference"])
    if kind == "op":
        g = _grid(rng, 18, 200)
        return dict(kind=kind, **g, pml=4, adjoint=rng.random() < 0.5)
    if kind == "prec":
        g = _grid(rng, 18, 96)
        return dict(kind=kind, **g, pml=4, zt=rng.choice(["fft", "eigen"]), adjoint=rng.random() < 0.5)
    if kind == "prec_batch":
        g = _grid(rng, 24, 128)
        return dict(kind=kind, **g, pml=6, zt="fft", nrhs=rng.randint(2, 16))
    if kind == "solve":
        if rng.random() < 0.3:
            g = _grid(rng, 20, 64)
            return dict(kind=kind, **g, pml=4, prec="c128", zt="fft", nrhs=1, medium="homogeneous", restart=20,
                        tol=1e-8)
        g = _grid(rng, 20, 128)
        return dict(kind=kind, **g, pml=4, prec="c64", zt="eigen", nrhs=rng.randint(1, 8), medium="layered",
                    restart=20, tol=1e-9)
    if kind == "step":
        g = _grid(rng, 32, 190)
        return dict(kind=kind, **g, pml=8, prec="c64", zt="eigen", nrhs=rng.randint(1, 4), medium="layered",
                    restart=20, tol=1e-9)
    if kind == "group":
        g = _grid(rng, 48, 112)
        return dict(kind=kind, **g, pml=8, grids=rng.randint(2, 4), nrhs=rng.randint(1, 2), restart=20, tol=1e-9)
    if kind == "gradient":
        g = _grid(rng, 40, 96)
        return dict(kind=kind, **g, pml=8, nrhs=rng.randint(1, 8), nrecv=rng.randint(4, 20), restart=30, tol=1e-10)
    n = _side(rng, 10, 50)
    return dict(kind=kind, nx=n + 8, ny=n + 8, nz=n + 8, pml=4, spg=4, restart=30, tol=1e-10)


# ------------------------------------------------------------------ inputs
def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _problem(case, seed, nsrc, medium="layered", shape=None):
    nx, ny, nz = shape or (case["nx"], case["ny"], case["nz"])
    p = media.layered_medium(nx, ny, nz, 10.0, case["pml"], seed, ppw=8.0, n_sources=nsrc)
    if medium == "homogeneous":
        c = 1500.0
        p.omega = 2.0 * math.pi * c / (10.0 * p.h)
        p.s2 = np.full(p.shape, 1.0 / (c * c))
    return p


def _tensors(p, nsrc):
    s2 = torch.from_numpy(np.ascontiguousarray(p.s2)).to(_dev())
    f = torch.stack([torch.from_numpy(p.rhs(i)).to(_dev()) for i in range(nsrc)]) if nsrc else None
    return s2, f


def _solver(p, s2, prec, zt, restart=20, tol=1e-8):
    g = helm3d.grid_mode_n(p.nx, p.ny, p.nz, p.h, p.pml, p.omega)
    o = helm3d.default_opts(precision=helm3d.PREC_C64 if prec == "c64" else helm3d.PREC_C128, restart=restart, tol=tol,
                            beta_prec=BETA[zt], max_iter=20000, device=_dev().index,
                            z_transform=helm3d.ZT_PML_EIGEN if zt == "eigen" else helm3d.ZT_FFT)
    return helm3d.Solver(g, s2, o)


def _random(shape, seed):
    gen = torch.Generator(device=_dev())
    gen.manual_seed(seed)
    return torch.randn(shape, generator=gen, dtype=torch.complex128, device=_dev())


def _group_shapes(case):
    """The case's own grid and up to three uneven ones around it (the
    benchmark's uneven sides: 48..112)."""
    return [(case["nx"], case["ny"], case["nz"]), (48, 48, 48), (64, 80, 72), (56, 48, 56)][:case["grids"]]


def _reference_problem(case, seed):
    """The reference's grid (PML in x and y, sponge in z, 3200 m) with a
    smooth heterogeneous medium, and a point source in its interior."""
    pml, spg = case["pml"], case["spg"]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    npx = nx - 2 * pml
    h = (LEN_REF + 2.0 * pml * LEN_REF / npx) / nx
    npz = nz - 2 * spg
    lz = LEN_REF + 2.0 * spg * LEN_REF / npz
    hz = lz / nz
    rng = np.random.RandomState(seed % (1 << 31))
    x, y, z = (np.arange(n, dtype=np.float64) / n for n in (nx, ny, nz))
    ph = rng.uniform(0.0, 2 * math.pi, 3)
    bump = np.cos(2 * math.pi * x + ph[0])[None, None, :] * np.cos(2 * math.pi * y + ph[1])[None, :, None] * \
        np.cos(2 * math.pi * z + ph[2])[:, None, None]
    s2 = 1.0 / (C_REF * (1.0 + 0.03 * bump)) ** 2
    f = np.zeros((nz, ny, nx), dtype=np.complex128)
    f[rng.randint(spg + 2, nz - spg - 2), rng.randint(pml + 2, ny - pml - 2),
      rng.randint(pml + 2, nx - pml - 2)] = -1.0 / (h * h * hz)
    return h, hz, lz, s2, f


def prepare(case, seed):
    kind, seed = case["kind"], int(seed)
    if kind in ("op", "prec", "prec_batch"):
        p = _problem(case, seed, 0)
        s2, _ = _tensors(p, 0)
        prec = "c64" if kind == "prec_batch" else "c128"
        if kind == "op":
            # the operator does not use the preconditioner: the cheaper one
            prec = "c64"
        s = _solver(p, s2, prec, case.get("zt", "fft"))
        x = _random(((case["nrhs"],) if kind == "prec_batch" else ()) + p.shape, seed)
        return dict(case=case, solver=s, x=x)
    if kind in ("solve", "step"):
        p = _problem(case, seed, case["nrhs"], case["medium"])
        s2, f = _tensors(p, case["nrhs"])
        s = _solver(p, s2, case["prec"], case["zt"], case["restart"], case["tol"])
        return dict(case=case, solver=s, s2=s2, f=f, u=torch.empty_like(f))
    if kind == "group":
        ss, s2s, fs, us = [], [], [], []
        for q, shape in enumerate(_group_shapes(case)):
            p = _problem(case, seed + 1000 * q, case["nrhs"], shape=shape)
            s2, f = _tensors(p, case["nrhs"])
            ss.append(_solver(p, s2, "c64", "eigen", case["restart"], case["tol"]))
            s2s.append(s2)
            fs.append(f)
            us.append(torch.empty_like(f))
        return dict(case=case, solvers=ss, s2=s2s, f=fs, u=us)
    if kind == "gradient":
        p, recv, data = _gradient_problem(case, seed)
        s2, f = _tensors(p, case["nrhs"])
        s = _solver(p, s2, "c64", "eigen", case["restart"], case["tol"])
        return dict(case=case, solver=s, f=f, recv=torch.from_numpy(recv).to(_dev()), data=data)
    h, hz, lz, s2, f = _reference_problem(case, seed)
    g = helm3d.grid_mode_r(case["nx"], case["ny"], case["nz"], h, hz, case["pml"], case["spg"], lz,
                           2.0 * math.pi * HZ_REF)
    o = helm3d.default_opts(mode=helm3d.MODE_R, precision=helm3d.PREC_C128, kz_symbol=helm3d.KZ_REFERENCE,
                            beta_prec=0.5, quirk_q1=1, restart=case["restart"], max_iter=5000, tol=case["tol"],
                            device=_dev().index)
    s = helm3d.Solver(g, torch.from_numpy(s2).to(_dev()), o)
    return dict(case=case, solver=s, f=torch.from_numpy(f).to(_dev()))


def _gradient_problem(case, seed):
    """A smooth starting model, receivers on the plane below the top PML and
    observed data of the size the wavefield has there."""
    p = _problem(case, seed, case["nrhs"])
    nx, nz, m = p.nx, p.nz, case["nrecv"]
    xi = np.linspace(p.pml + 1, nx - 2 - p.pml, m).round().astype(np.int64)
    zi = np.linspace(p.pml + 1, nz - 2 - p.pml, m).round().astype(np.int64)
    kk, ii = np.meshgrid(zi, xi, indexing="ij")
    recv = ((kk * p.ny + p.pml + 2) * nx + ii).ravel().astype(np.int64)
    scale = 1.0 / (4.0 * math.pi * 0.3 * p.h * nx)
    data = scale * _random((case["nrhs"], recv.size), seed + 1)
    return p, recv, data


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "op":
        s = state["solver"]
        return s.apply_op_adjoint(state["x"]) if case["adjoint"] else s.apply_op(state["x"])
    if kind == "prec":
        s = state["solver"]
        return s.apply_prec_adjoint(state["x"]) if case["adjoint"] else s.apply_prec(state["x"])
    if kind == "prec_batch":
        # a complex64 preconditioner's output, kept in its own precision
        return state["solver"].apply_prec_batch(state["x"]).to(torch.complex64)
    if kind == "solve":
        return state["solver"].solve(state["f"], nrhs=case["nrhs"], u=state["u"])
    if kind == "step":
        return state["solver"].solve_medium(state["s2"], state["f"], nrhs=case["nrhs"], u=state["u"])
    if kind == "group":
        for s, s2 in zip(state["solvers"], state["s2"]):
            s.set_medium(s2)
        return helm3d.solve_group(state["solvers"], state["f"], us=state["u"])
    if kind == "gradient":
        J, grad = state["solver"].misfit_grad(state["f"], state["recv"], state["data"])
        return {"misfit": J, "grad": grad}
    return state["solver"].solve(state["f"])


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: the inputs once, the outputs once and, where the pass uses a
    factor that it did not make, the factor once per application.
    Operations: 8 nx^2 per grid point for a factor (an explicit inverse of
    every block), 32 nx per point and vector for a sweep (two block products
    per line), 64 per point and vector for the operator; a nominal number of
    applications for a solve."""
    kind = case["kind"]
    n = case["nx"] * case["ny"] * case["nz"]
    nx = case["nx"]
    if kind == "op":
        return {"bytes": 40.0 * n, "flops": 64.0 * n}
    e = 8 if case.get("prec", "c128") == "c64" or kind in ("prec_batch", "step", "group", "gradient") else 16
    factor, sweep = 8.0 * nx * nx * n, 32.0 * nx * n
    if kind == "prec":
        return {"bytes": 32.0 * n + e * nx * n, "flops": sweep}
    r = case.get("nrhs", 1)
    if kind == "prec_batch":
        return {"bytes": 24.0 * n * r + e * nx * n, "flops": sweep * r}
    per = sweep + 64.0 * n
    if kind == "solve":
        its = 10 if case["zt"] == "eigen" else 240
        return {"bytes": 32.0 * n * r + e * nx * n * its, "flops": per * r * its}
    if kind == "step":
        return {"bytes": (8.0 + 32.0 * r) * n + e * nx * n, "flops": factor + per * r * 8}
    if kind == "group":
        b = f = 0.0
        for gx, gy, gz in _group_shapes(case):
            m = gx * gy * gz
            b += (8.0 + 32.0 * r) * m + e * gx * m
            f += 8.0 * gx * gx * m + (32.0 * gx + 64.0) * m * r * 10
        return {"bytes": b, "flops": f}
    if kind == "gradient":
        its = 20
        return {"bytes": (16.0 * r + 8.0) * n + e * nx * n * its, "flops": per * r * its}
    its = 40
    return {"bytes": 32.0 * n + e * nx * n * its, "flops": sweep * its}


# ------------------------------------------------------- outputs in 64 bits
def _alpha(n, pml, i, omega):
    if pml == 0:
        return 1.0 + 0.0j
    if i < pml or i >= n - pml:
        x = 1.0 - i / pml if i < pml else 1.0 + (i - n + 1) / pml
        return -1j * omega / (1000.0 * x * x - 1j * omega)
    return 1.0 + 0.0j


def _couplings(n, pml, h, omega):
    """Coefficients of u[i-1] and u[i+1] of the PML-stretched second difference."""
    a = [_alpha(n, pml, float(i), omega) for i in range(n)]
    cm = [a[i] * _alpha(n, pml, i - 0.5, omega) / (h * h) for i in range(n)]
    cp = [a[i] * _alpha(n, pml, i + 0.5, omega) / (h * h) for i in range(n)]
    return tuple(torch.tensor(v, dtype=torch.complex128, device=_dev()) for v in (cm, cp))


def _tridiag(cm, cp):
    return torch.diag(-(cm + cp)) + torch.diag(cm[1:], -1) + torch.diag(cp[:-1], 1)


class _Blocks:
    """The 2D systems of every z mode, block tridiagonal over y, by block
    elimination: sub[j] u_{j-1} + D_j u_j + sup[j] u_{j+1} = f_j."""

    def __init__(self, sub, D, sup):
        self.sub, self.sup, self.G = sub, sup, []
        for j in range(len(sub)):
            S = D(j)
            if j:
                S = S - sub[j] * sup[j - 1] * self.G[-1]
            self.G.append(torch.linalg.inv(S))

    def solve(self, f):
        """f: (modes, ny, nx, vectors)."""
        ny, y = len(self.G), torch.empty_like(f)
        for j in range(ny):
            y[:, j] = self.G[j] @ (f[:, j] - self.sub[j] * y[:, j - 1] if j else f[:, j])
        for j in range(ny - 2, -1, -1):
            y[:, j] -= self.sup[j] * (self.G[j] @ y[:, j + 1])
        return y


class _Exact:
    """The mode N operator A, the preconditioner M and A u = f in complex128.
    Vectors: (vectors, nz, ny, nx)."""

    def __init__(self, p, s2, zt, beta, adjoint=False, factor=True):
        self.p, self.s2, self.adj = p, s2, adjoint
        self.c = [_couplings(n, p.pml, p.h, p.omega) for n in (p.nx, p.ny, p.nz)]
        self.w2 = p.omega * p.omega
        if factor:
            self._factor(zt, beta)

    def op(self, u):
        conj = (lambda t: t.conj()) if self.adj else (lambda t: t)
        out = self.w2 * self.s2 * u
        for axis, (cm, cp) in zip((3, 2, 1), self.c):
            shape = [1, 1, 1, 1]
            shape[axis] = -1
            n = u.shape[axis]
            out -= conj(cm + cp).reshape(shape) * u
            lo, hi = u.narrow(axis, 0, n - 1), u.narrow(axis, 1, n - 1)
            # rows 1.. take the lower neighbour, rows ..n-2 the upper one
            dn, up = (cp[:-1], cm[1:]) if self.adj else (cm[1:], cp[:-1])
            out.narrow(axis, 1, n - 1).add_(conj(dn).reshape(shape) * lo)
            out.narrow(axis, 0, n - 1).add_(conj(up).reshape(shape) * hi)
        return out

    def _factor(self, zt, beta):
        p = self.p
        (cmx, cpx), (cmy, cpy), (cmz, cpz) = self.c
        lo, hi = (p.pml, p.nz - p.pml) if p.nz > 2 * p.pml else (0, p.nz)
        base = self.w2 * self.s2[lo:hi].mean(0) * (1.0 + 1j * beta)
        if zt == "eigen":
            lam, W = torch.linalg.eig(_tridiag(cmz, cpz).cpu())
            lam, W = lam.to(_dev()), W.to(_dev())
            Wi = torch.linalg.inv(W)
        else:
            k = torch.arange(p.nz, device=_dev(), dtype=torch.float64)
            lam = -(4.0 / (p.h * p.h)) * torch.sin(math.pi * k / p.nz) ** 2 + 0j
            jk = torch.outer(k, k)
            F = torch.exp(-2j * math.pi * torch.remainder(jk, p.nz) / p.nz)
            Wi, W = F, F.conj() / p.nz
        Tx, eye = _tridiag(cmx, cpx), torch.eye(p.nx, dtype=torch.complex128, device=_dev())
        sub, sup = cmy, cpy
        if self.adj:
            sub, sup = torch.cat([cpy[-1:], cpy[:-1]]).conj(), torch.cat([cmy[1:], cmy[:1]]).conj()

        def D(j):
            d = Tx + torch.diag(base[j] - cmy[j] - cpy[j])
            m = d + lam[:, None, None] * eye
            return m.mH if self.adj else m
        self.blocks = _Blocks(sub.tolist(), D, sup.tolist())
        self.fwd, self.inv = (W.mH, Wi.mH) if self.adj else (Wi, W)

    def prec(self, x):
        R, nz, ny, nx = x.shape
        t = (self.fwd @ x.permute(1, 2, 3, 0).reshape(nz, -1)).reshape(nz, ny, nx, R)
        t = self.blocks.solve(t)
        return (self.inv @ t.reshape(nz, -1)).reshape(nz, ny, nx, R).permute(3, 0, 1, 2).contiguous()

    def solve(self, f):
        return torch.stack([_gmres(self.op, self.prec, f[r:r + 1])[0] for r in range(f.shape[0])])


def _gmres(A, M, f, tol=2e-14, m=40, cycles=6):
    """A u = f by right-preconditioned GMRES in complex128 (Gram-Schmidt twice)."""
    u, nf = torch.zeros_like(f), torch.linalg.vector_norm(f)
    best = None
    for _ in range(cycles):
        r = f - A(u)
        beta = torch.linalg.vector_norm(r)
        if best is not None and float(beta) > 0.5 * best:
            break
        best = float(beta)
        V = [(r / beta).reshape(-1)]
        H = torch.zeros((m + 1, m), dtype=torch.complex128)
        for j in range(m):
            w = A(M(V[j].reshape(f.shape))).reshape(-1)
            for _ in range(2):
                for i, v in enumerate(V):
                    h = torch.vdot(v, w)
                    w = w - h * v
                    H[i, j] += h.cpu()
            H[j + 1, j] = torch.linalg.vector_norm(w).cpu()
            V.append(w / H[j + 1, j].real)
            e = torch.zeros(j + 2, 1, dtype=torch.complex128)
            e[0] = beta.cpu()
            y = torch.linalg.lstsq(H[:j + 2, :j + 1], e).solution
            if float(torch.linalg.vector_norm(H[:j + 2, :j + 1] @ y - e)) <= tol * float(nf):
                break
        z = sum(v * complex(c) for v, c in zip(V, y[:, 0].tolist()))
        u = u + M(z.reshape(f.shape))
    return u


def _exact_reference(case, seed):
    h, hz, lz, s2, f = _reference_problem(case, seed)
    nx, ny, nz, pml, spg, beta = case["nx"], case["ny"], case["nz"], case["pml"], case["spg"], 0.5
    w = 2.0 * math.pi * HZ_REF
    # the 2D medium: the mean over the z range without its sponge, the
    # reference's running sum carried from one column to the next
    col, s0, acc = s2[spg:nz - spg].sum(0), np.zeros((ny, nx)), 0.0
    for j in range(pml, ny - pml):
        for i in range(pml, nx - pml):
            acc = (acc + col[j, i]) / (nz - 2 * spg)
            s0[j, i] = acc
    s0[:, :pml], s0[:, nx - pml:] = s0[:, pml:pml + 1], s0[:, nx - pml - 1:nx - pml]
    s0[:pml], s0[ny - pml:] = s0[pml:pml + 1], s0[ny - pml - 1:ny - pml]
    # dL with its Gaussian taper into the sponges
    dl = w * w * ((1.0 + 1j * beta) * s0 - s2)
    for k in range(nz):
        if k < spg or k > nz - spg:
            edge = spg if k < spg else nz - spg
            width = spg * hz if k < spg else lz - edge * hz
            dl[k] = w * w * ((1.0 + 1j * beta) * s0 - s2[edge]) * math.exp(-((k - edge) * hz / width / 0.3) ** 2)
    dl = torch.from_numpy(dl).to(_dev())
    k = np.arange(nz)
    kk = np.where(k < nz // 2 - 1, k, nz - k)
    lam = torch.from_numpy(-(2.0 * math.pi * kk / lz) ** 2 + 0j).to(_dev())
    (cmx, cpx), (cmy, cpy) = _couplings(nx, pml, h, w), _couplings(ny, pml, h, w)
    Tx, eye = _tridiag(cmx, cpx), torch.eye(nx, dtype=torch.complex128, device=_dev())
    base = torch.from_numpy(w * w * s0 * (1.0 + 1j * beta)).to(_dev())
    b = _Blocks(cmy.tolist(), lambda j: Tx + torch.diag(base[j] - cmy[j] - cpy[j]) + lam[:, None, None] * eye,
                cpy.tolist())

    def l0inv(x):
        return torch.fft.ifft(b.solve(torch.fft.fft(x[0], dim=0)[..., None])[..., 0], dim=0)[None]
    f = torch.from_numpy(f).to(_dev())[None]
    return l0inv(_gmres(lambda x: x - dl * l0inv(x), lambda x: x, f, m=60))[0]


def exact(case, seed):
    kind, seed = case["kind"], int(seed)
    if case["nx"] > 160:
        # the complex128 blocks of the largest grids take minutes to invert here
        if kind != "op":
            return None
    if kind == "op":
        p = _problem(case, seed, 0)
        s2, _ = _tensors(p, 0)
        return _Exact(p, s2, "fft", 0.0, case["adjoint"], factor=False).op(_random(p.shape, seed)[None])[0]
    if kind in ("prec", "prec_batch"):
        p = _problem(case, seed, 0)
        s2, _ = _tensors(p, 0)
        x = _random(((case["nrhs"],) if kind == "prec_batch" else (1,)) + p.shape, seed)
        if kind == "prec":
            x = _random(p.shape, seed)[None]
        y = _Exact(p, s2, case["zt"], BETA[case["zt"]], case.get("adjoint", False)).prec(x)
        return y if kind == "prec_batch" else y[0]
    if kind in ("solve", "step"):
        p = _problem(case, seed, case["nrhs"], case["medium"])
        s2, f = _tensors(p, case["nrhs"])
        return _Exact(p, s2, "eigen", 0.0).solve(f)
    if kind == "group":
        out = []
        for q, shape in enumerate(_group_shapes(case)):
            p = _problem(case, seed + 1000 * q, case["nrhs"], shape=shape)
            s2, f = _tensors(p, case["nrhs"])
            out.append(_Exact(p, s2, "eigen", 0.0).solve(f))
        return out
    if kind == "gradient":
        p, recv, data = _gradient_problem(case, seed)
        s2, f = _tensors(p, case["nrhs"])
        recv = torch.from_numpy(recv).to(_dev())
        u = _Exact(p, s2, "eigen", 0.0).solve(f)
        r = u.reshape(case["nrhs"], -1)[:, recv] - data
        g = torch.zeros_like(u)
        for q in range(case["nrhs"]):
            g[q].view(-1).index_add_(0, recv, -r[q])
        lam = _Exact(p, s2, "eigen", 0.0, adjoint=True).solve(g)
        grad = (lam.conj() * u).real.sum(0) * (p.omega * p.omega)
        return {"misfit": 0.5 * float((r.abs() ** 2).sum()), "grad": grad}
    return _exact_reference(case, seed)
