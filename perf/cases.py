"""Workloads of the time-step library, as a host program calls it.

Two kinds of call, both through the public entry points:

  run      a restart state is uploaded (tbl_upload_state), the box is advanced
           `steps` time steps (tbl_step) and u, v, w, p and the GMRES warm
           start p' come back (tbl_download_state) into the caller's pinned
           buffers: the life of the reference program between two restart files.
  adjoint  the same upload, a recorded window of `steps` steps
           (tbl_forward_window) and its discrete adjoint (tbl_backward_window):
           the objective, dL/dc of the wall control and dL/d(initial state).

Every pass starts from the same uploaded state, so every pass does the same
steps.  The states are a 1/7-law boundary layer with a seeded, divergence-free
perturbation, past the start of the recycling (the inflow is rescaled every
step, as it is in all but the first steps of a run).
"""
import ctypes as C
import math

import numpy as np
import torch

from turbulentbl_gb300 import abi
from turbulentbl_gb300.lib import TblGpu
from turbulentbl_gb300.mesh import RunParams, make_mesh, recycle_plane
from turbulentbl_gb300.synth import THETA0, rescaling_state

FIELDS = ("u", "v", "w", "p", "pcorr")
NSTEP0 = 2000          # steps the run has behind it: past every program's recycling start
PATCH = (0.25, 0.75)   # streamwise extent of the adjoint's wall-shear patch, as a fraction of the box
D = torch.float64
FAST = abi.TBL_FLAG_RB_ORDER | abi.TBL_FLAG_SSOR_SPAN_BLOCKS | abi.TBL_FLAG_SSOR_STREAM_BLOCKS


def _case(name, nx, nyw, nzs, lx, lyw, lzs, beta, re_theta, nproc, kmax, tol, steps, kind="run", mixed=False,
          variant=0, fast=False, ckpt=0):
    """nx streamwise, nyw wall-normal, nzs span points; lengths, stretching and
    Reynolds number of the box; nproc slabs; GMRES restart and tolerance."""
    return dict(name=name, kind=kind, nx=nx, nyw=nyw, nzs=nzs, lx=lx, lyw=lyw, lzs=lzs, beta=beta,
                re_theta=re_theta, nproc=nproc, kmax=kmax, tol=tol, steps=steps, mixed=mixed, variant=variant,
                fast=fast, ckpt=ckpt)


def listed():
    return [
        # the sizes of the tests and of a first run of a new set-up: a step is launches and latency
        _case("tiny_fp64", 32, 24, 16, 5.0, 3.0, 1.0, 2.0, 300.0, 2, 20, 1e-8, 5),
        # the 128 x 64 x 64 box with its own solver settings, one whole recycling window (5 steps, one rescaling)
        _case("box128_fp64", 128, 64, 64, 20.0, 3.0, 4.0, 2.0, 300.0, 8, 30, 1e-8, 5),
        # the same box in mixed precision
        _case("box128_mixed", 128, 64, 64, 20.0, 3.0, 4.0, 2.0, 300.0, 8, 30, 1e-10, 5, mixed=True),
        # a grid with no round sizes and an odd span, the originalTBL program (no upper Peclet bound, inflow ramp)
        _case("ragged_original_fp64", 201, 59, 75, 30.0, 3.0, 4.5, 2.0, 300.0, 5, 25, 1e-9, 3, variant=1),
        # the dnssetbl program: its slab partition (remainder on the last ranks), central span rows, scaled v inflow
        _case("dnssetbl_fp64", 160, 81, 64, 24.0, 3.0, 4.0, 2.0, 300.0, 7, 30, 1e-8, 3, variant=2),
        # a ragged grid in mixed precision, slabs that do not divide the planes
        _case("ragged_mixed", 333, 85, 97, 45.0, 3.0, 5.0, 2.1, 300.0, 6, 40, 1e-10, 2, mixed=True),
        # the throughput options (red-black diffusion, span and streamwise SSOR blocks) in FP64
        _case("box256_fast_fp64", 256, 96, 96, 20.0, 3.0, 4.0, 2.0, 300.0, 8, 30, 1e-10, 2, fast=True),
        # the headline box, 512 x 128 x 128, FP64: what a production run spends its time on
        _case("box512_fp64", 512, 128, 128, 40.0, 3.0, 6.0, 2.2, 300.0, 8, 40, 1e-10, 1),
        # the headline box in mixed precision
        _case("box512_mixed", 512, 128, 128, 40.0, 3.0, 6.0, 2.2, 300.0, 8, 40, 1e-10, 1, mixed=True),
        # the headline box with the throughput options in mixed precision: the fastest way to run it
        _case("box512_fast_mixed", 512, 128, 128, 40.0, 3.0, 6.0, 2.2, 300.0, 8, 40, 1e-10, 1, mixed=True, fast=True),
        # the largest: towards the 1024 x 192 x 256 box (its stretching, Reynolds number and restart length)
        _case("large_mixed", 768, 144, 192, 45.0, 3.5, 6.0, 2.4, 400.0, 8, 30, 1e-10, 1, mixed=True),
        # gradient of the wall shear with respect to the wall control over a window with one recomputed segment
        _case("adjoint128", 128, 64, 64, 20.0, 3.0, 4.0, 2.0, 300.0, 8, 30, 1e-10, 4, kind="adjoint", ckpt=2),
    ]


def draw(rng):
    """Sizes spread over the logarithm of the points, from the tests' grids to
    the headline box (mixed precision and the throughput options included)."""
    kind = rng.choice(["fp64", "fp64", "mixed", "mixed", "fast", "adjoint"])
    top = 8.4e6 if kind in ("fp64", "mixed") else 2.5e6 if kind == "fast" else 5e5
    points = math.exp(rng.uniform(math.log(1.2e4), math.log(top)))
    # streamwise : wall-normal : span about 4 : 1 : 1, each off by up to a third
    s = (points / 4.0) ** (1.0 / 3.0)
    nx = max(24, int(4.0 * s * rng.uniform(0.67, 1.33)))
    nyw = min(150, max(20, int(s * rng.uniform(0.75, 1.33))))
    nzs = max(12, int(points / (nx * nyw)))
    if kind == "fast":
        nzs += nzs % 2  # the red-black colouring needs an even span
    nproc = rng.randint(1, max(1, min(8, (nyw - 1) // 4)))
    steps = 1 if points > 1e6 else rng.randint(1, 3)
    mixed = kind == "mixed" or (kind == "fast" and rng.random() < 0.5)
    adj = kind == "adjoint"
    c = _case("", nx, nyw, nzs, nx * 20.0 / 128 * rng.uniform(0.8, 1.1), 3.0, nzs * rng.uniform(0.045, 0.065),
              rng.uniform(1.8, 2.2), rng.uniform(250.0, 400.0), nproc, rng.randint(15, 40),
              1e-10 if mixed or adj else rng.choice([1e-8, 1e-9, 1e-10]), steps + 1 if adj else steps,
              kind="adjoint" if adj else "run", mixed=mixed,
              variant=rng.choice([0, 0, 1, 2]) if kind in ("fp64", "mixed") else 0, fast=kind == "fast",
              ckpt=rng.randint(1, 2) if adj else 0)
    del c["name"]
    return c


# ------------------------------------------------------------------- inputs
def _grid(case):
    return case["nx"], case["nzs"] + 2, case["nyw"]


def _smooth(shape, gen, width=2.0):
    """Gaussian noise smoothed over `width` cells, periodic, on the GPU."""
    f = torch.fft.rfftn(torch.randn(shape, generator=gen, device="cuda", dtype=D))
    for d, n in enumerate(shape):
        k = (torch.fft.rfftfreq if d == len(shape) - 1 else torch.fft.fftfreq)(n, device="cuda", dtype=D)
        f = f * torch.exp(-2.0 * (math.pi * width * k) ** 2).view([-1 if q == d else 1 for q in range(len(shape))])
    return torch.fft.irfftn(f, s=shape)


def _velocity(case, mesh, seed):
    """u, v, w on the GPU as (nz, ny, nx): the mean profile and the curl of a
    seeded vector potential that vanishes at the wall."""
    nx, ny, nz = _grid(case)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    x3 = torch.tensor(mesh.x3, dtype=D, device="cuda")
    jac = torch.tensor(mesh.jac, dtype=D, device="cuda").view(-1, 1, 1)
    damp = (x3 ** 2 * torch.exp(-x3 ** 2)).view(-1, 1, 1)
    A = [_smooth((nz, ny - 2, nx), gen) * damp for _ in range(3)]
    dx = lambda f: torch.gradient(f, spacing=mesh.dx, dim=2)[0]
    dy = lambda f: (torch.roll(f, -1, 1) - torch.roll(f, 1, 1)) / (2.0 * mesh.dy)
    dz = lambda f: torch.gradient(f, spacing=mesh.dxi, dim=0)[0] / jac
    w3 = [dy(A[2]) - dz(A[1]), dz(A[0]) - dx(A[2]), dx(A[1]) - dy(A[0])]
    rms = torch.sqrt(sum((q * q).mean() for q in w3) / 3.0)
    mean = torch.clamp(torch.clamp(x3, min=0.0) ** (1.0 / 7.0), max=1.0).view(-1, 1, 1)
    out = []
    for q, f in enumerate(w3):
        f = 0.05 / rms * f + (mean if q == 0 else 0.0)
        f[0] = 0.0
        out.append(torch.cat([f[:, -1:], f, f[:, :1]], dim=1))
    return out


def _host(t):
    """A (nx, ny, nz) column-major view of a pinned host copy of t (nz, ny, nx)."""
    h = torch.empty(t.shape, dtype=D, pin_memory=True)
    h.copy_(t)
    return h.numpy().T


def _problem(case, seed):
    """Mesh, run parameters and restart state (numpy, column-major)."""
    nx, ny, nz = _grid(case)
    mesh = make_mesh(nx, ny, nz, case["lx"], case["lzs"], case["lyw"], case["beta"])
    U = _velocity(case, mesh, seed)
    h = np.diff(mesh.x3)
    hz = torch.tensor(np.minimum(np.r_[h[0], h], np.r_[h, h[-1]]), dtype=D, device="cuda").view(-1, 1, 1)
    s = U[0].abs() / mesh.dx + U[1].abs() / mesh.dy + U[2].abs() / hz
    dt = 0.3 / float(s[1:-1, 1:-1, 1:-1].max())
    rp = RunParams(dt=dt, re=case["re_theta"] / THETA0, ue=1.0, nproc=case["nproc"], irec=recycle_plane(nx),
                   kmax=case["kmax"], errtol=case["tol"], precision=abi.TBL_PREC_MIXED if case["mixed"] else 0,
                   mixed_kmax=case["kmax"], mixed_outer_tol=case["tol"], flags=FAST if case["fast"] else 0)
    rp.use_variant(case["variant"])
    if case["kind"] == "adjoint":
        rp.cum = 1000  # the recycling means stay fixed over a window
    means = [np.asfortranarray(u[:, 1:-1].mean(1).cpu().numpy().T) for u in U]
    bl, wt, newk, ksep = rescaling_state(means[0], mesh.x3, 1.0, rp.irec)
    st = dict(zip(("u", "v", "w"), map(_host, U)))
    for f in ("p", "pcorr"):
        st[f] = _host(torch.zeros((nz, ny, nx), dtype=D))
    st.update(zip(("usum2", "vsum2", "wsum2"), means))
    st.update(wt=np.asfortranarray(wt), newk=newk, bltkns=bl, ksep=ksep, lamda=1.0, time=0.0, nstep=NSTEP0, cont=0,
              cnt2=NSTEP0, ume1=np.minimum(np.maximum(mesh.x3, 0.0) ** (1.0 / 7.0), 1.0))
    return mesh, rp, st


def _control(case, seed):
    """A small smooth blowing/suction profile of the wall, (nx, ny-2)."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    c = _smooth((case["nzs"], case["nx"]), gen)
    return np.asfortranarray((1e-3 / c.std() * c).cpu().numpy().T)


def prepare(case, seed):
    mesh, rp, st = _problem(case, seed)
    s = dict(case=case, gpu=TblGpu(mesh, rp), state=st)
    if case["kind"] == "adjoint":
        s["gpu"].set_wall_control(_control(case, seed))
        s["patch"] = tuple(f * case["lx"] for f in PATCH)
        # the tape of a window belongs to the handle: a program that improves a control runs many windows on it
        s["gpu"].upload(st)
        s["gpu"].forward_window(case["steps"], *s["patch"], case["ckpt"])
        return s
    nx, ny, nz = _grid(case)
    s["out"] = {f: torch.zeros((nz, ny, nx), dtype=D, pin_memory=True) for f in FIELDS}
    s["into"] = abi.TblState()
    for f in FIELDS:
        setattr(s["into"], f, abi.dptr(s["out"][f].numpy()))
    return s


# --------------------------------------------------------------------- a pass
def run(s):
    case, g = s["case"], s["gpu"]
    g.upload(s["state"])
    if case["kind"] == "adjoint":
        J, _ = g.forward_window(case["steps"], *s["patch"], case["ckpt"])
        dc, d0, _ = g.backward_window(1.0, want_initial=True)
        return dict(J=J, dc=dc, **{"d" + f: d0[f] for f in ("u", "v", "w", "p")})
    g.step(case["steps"])
    st = g.lib.tbl_download_state(g._h, C.byref(s["into"]))
    if st != abi.TBL_OK:
        raise RuntimeError("tbl_download_state: %d" % st)
    if case["mixed"]:  # single-precision fields, and p' to the refinement's 1e-8: their own type
        return {f: t.float() for f, t in s["out"].items()}
    return s["out"]


def work(case):
    """The state read and written once, and the operations of one application
    of each operator of a step (convection, diffusion, divergence, Poisson,
    projection): a step cannot do with less, however its systems are solved."""
    nx, ny, nz = _grid(case)
    n = nx * ny * nz
    w = 4 if case["mixed"] else 8
    sweeps = 1 if case["kind"] == "run" else 3  # a window's adjoint: forward, recomputation, transposed steps
    return {"bytes": float(n * (4 * w + 8) * 2), "flops": float(n * case["steps"] * sweeps * (120 + 3 * 15 + 12 + 15 + 20))}


# ------------------------------------------- the same call in plain 64-bit torch
# Arrays are (nz, ny, nx).  The implicit diffusion and the pressure-Poisson
# system are solved directly: sine transform along x, Fourier along the
# periodic span, eigenvectors of the (symmetrised) wall-normal operator.
class _Exact:
    def __init__(self, case, mesh, rp, st):
        self.c, self.m, self.rp = case, mesh, rp
        self.nx, self.ny, self.nz = _grid(case)
        T = lambda a: torch.tensor(np.asarray(a), dtype=D, device="cuda")
        self.x3, self.jinv, self.j2 = T(mesh.x3), T(1.0 / mesh.jac), T(mesh.jac2)
        a = (self.jinv / mesh.dxi) ** 2
        b = self.j2 / (2.0 * mesh.dxi) * self.jinv ** 3
        self.ab, self.at = (a + b)[1:-1], (a - b)[1:-1]
        self.aw, self.as_ = 1.0 / mesh.dx ** 2, 1.0 / mesh.dy ** 2
        n = self.nx - 2
        q = torch.arange(1, n + 1, dtype=D, device="cuda")
        self.S = math.sqrt(2.0 / (n + 1)) * torch.sin(math.pi / (n + 1) * q[:, None] * q[None, :])
        lx = self.aw * (2.0 * torch.cos(math.pi * q / (n + 1)) - 2.0)
        J = self.ny - 2
        ly = self.as_ * (2.0 * torch.cos(2.0 * math.pi * torch.arange(J // 2 + 1, dtype=D, device="cuda") / J) - 2.0)
        off = torch.sqrt(self.at[:-1] * self.ab[1:])
        lz, self.Z = torch.linalg.eigh(torch.diag(-2.0 * a[1:-1]) + torch.diag(off, 1) + torch.diag(off, -1))
        self.e = torch.cumprod(torch.cat([torch.ones(1, dtype=D, device="cuda"), torch.sqrt(self.at[:-1] / self.ab[1:])]), 0)
        self.lam = lz[:, None, None] + ly[None, :, None] + lx[None, None, :]
        P, nz = rp.nproc, self.nz
        if case["variant"] == 2:
            size = [nz // P + (r >= P - nz % P) for r in range(P)]
            self.slab = np.repeat(np.arange(P), size)
        else:
            self.slab = np.minimum((np.arange(nz) - 1) // ((nz - 1) // P), P - 1)
        self.mean = [T(st[f].T) for f in ("usum2", "vsum2", "wsum2")]
        self.ume1, self.newk = T(st["ume1"]), np.asarray(st["newk"]) - 1
        self.nstep, self.ran = st["nstep"], 0

    def solve(self, f, shift, scale):
        """x with (shift + scale L7) x = f on the interior, zero around it."""
        f = torch.einsum("kl,kji->lji", self.Z, f * self.e[:, None, None])
        f = torch.fft.rfft(f @ self.S, dim=1) / (shift + scale * self.lam)
        f = torch.fft.irfft(f, n=self.ny - 2, dim=1) @ self.S
        return torch.einsum("kl,lji->kji", self.Z, f) / self.e[:, None, None]

    def ghosts(self, F):
        return torch.cat([F[:, -2:-1], F[:, 1:-1], F[:, 1:2]], 1)

    def inflow(self, U, live, file):
        ir, v = self.rp.irec - 1, self.c["variant"]
        eps = min((self.nstep if v == 2 else NSTEP0 + self.ran) * 5.0e-5, 1.0)
        rows = [[], [], []]
        for k in range(1, self.nz - 1):
            nk = self.newk[k]
            if self.mean[0][k, ir] < 0.99 * self.rp.ue:
                own = self.slab[k] == self.slab[nk] and 1 <= nk <= self.nz - 2
                mu = eps * self.mean[0][nk, ir] + (1 - eps) * self.ume1[k] if v else self.ume1[k]
                for q, mq in enumerate((mu, self.mean[1][nk, ir], self.mean[2][nk, ir])):
                    rows[q].append(mq + (live if own else file)[q][nk])
            else:
                for q in range(3):
                    rows[q].append(self.mean[q][k, ir].expand(self.ny - 2))
        out = []
        for F, r in zip(U, rows):
            F = F.clone()
            F[1:-1, 1:-1, 0] = torch.stack(r)
            out.append(F)
        return out

    def convection(self, U, F):
        """Convection of F by U at the interior points."""
        v, m = self.c["variant"], self.m
        win = (lambda Pe, hi: Pe.abs() > 2) if v == 2 else (lambda Pe, hi: Pe > 2) if v == 1 else (
            lambda Pe, hi: (Pe > 2) & (Pe < hi))
        tot = 0.0
        X = F[:, 1:-1]
        A = [u[1:-1, 1:-1, 1:-1] for u in U]
        z = self.x3
        for d, (h, hi) in enumerate(((m.dx, 50.0), (m.dy, 50.0), (m.dxi, 5.0))):
            a = A[d]
            if d == 1:
                W = X[1:-1, :, 1:-1]
                m2, m1, p1, p2 = (torch.roll(W, q, 1) for q in (2, 1, -1, -2))
            else:
                W = X[1:-1] if d == 0 else X[:, :, 1:-1]
                g = torch.nn.functional.pad(W, (1, 1) if d == 0 else (0, 0, 0, 0, 1, 1))
                n = W.shape[2 if d == 0 else 0] - 2
                m2, m1, p1, p2 = (g.narrow(2 if d == 0 else 0, q, n) for q in (0, 1, 3, 4))
                W = W.narrow(2 if d == 0 else 0, 1, n)
            hp = h if d < 2 else (z[2:] - z[1:-1]).view(-1, 1, 1)
            Pe = torch.where(a > -1.0, 1.0, -1.0) * self.rp.re * a.detach() * hp
            dis = a.abs() * (p2 - 4 * p1 + 6 * W - 4 * m1 + m2) * (0.25 / h)
            r = torch.where(win(Pe, hi), dis, 0.0) + a * (m2 - 8 * m1 + 8 * p1 - p2) / (12.0 * h)
            lim = a * (p1 - m1) / (2.0 * h)
            if d == 1 and v != 2:
                lim = torch.clamp(a, min=0.0) * (W - m1) / h + torch.clamp(a, max=0.0) * (p1 - W) / h
            dim = 2 - d
            n = r.shape[dim]
            r = torch.cat([lim.narrow(dim, 0, 1), r.narrow(dim, 1, n - 2), lim.narrow(dim, n - 1, 1)], dim)
            tot = tot + (r * self.jinv[1:-1].view(-1, 1, 1) if d == 2 else r)
        return tot

    def grad(self, P):
        m = self.m
        return (0.5 * (P[1:-1, 1:-1, 2:] - P[1:-1, 1:-1, :-2]) / m.dx,
                0.5 * (P[1:-1, 2:, 1:-1] - P[1:-1, :-2, 1:-1]) / m.dy,
                0.5 * (P[2:, 1:-1, 1:-1] - P[:-2, 1:-1, 1:-1]) * (self.jinv[1:-1].view(-1, 1, 1) / m.dxi))

    def inside(self, F, x):
        F = F.clone()
        F[1:-1, 1:-1, 1:-1] = x
        return F

    def step(self, U, P, live, file, c):
        m, rp, dt, re = self.m, self.rp, self.rp.dt, self.rp.re
        self.nstep += 1
        old = U[0][:, :, 0]
        U = self.inflow(U, live, file)  # the ghost rows follow at the end of the step only
        t = -dt / re
        g = self.grad(P)
        new = []
        for q, F in enumerate(U):
            f = F[1:-1, 1:-1, 1:-1] - dt * self.convection(U, F) - dt * g[q]
            e = torch.zeros_like(f)
            e[:, :, 0] += self.aw * F[1:-1, 1:-1, 0]
            e[:, :, -1] += self.aw * F[1:-1, 1:-1, -1]
            e[0] += self.ab[0] * F[0, 1:-1, 1:-1]
            e[-1] += self.at[-1] * F[-1, 1:-1, 1:-1]
            new.append(self.inside(F, self.solve(f - t * e, 1.0, t)))
        U = new
        u, v, w = U[0], self.ghosts(U[1]), U[2]
        zz = (self.x3[2:] - self.x3[:-2]).view(-1, 1, 1)
        div = (0.5 * (u[1:-1, 1:-1, 2:] - u[1:-1, 1:-1, :-2]) / m.dx + 0.5 * (v[1:-1, 2:, 1:-1] - v[1:-1, :-2, 1:-1]) / m.dy +
               (w[2:, 1:-1, 1:-1] - w[:-2, 1:-1, 1:-1]) / zz)
        C = self.inside(torch.zeros_like(P), self.solve(div / dt, 0.0, 1.0))
        I = slice(1, -1)
        C[0, I] = (4.0 * C[1, I] - C[2, I]) / 3.0
        C[-1, I] = (5.0 * C[-2, I] - 4.0 * C[-3, I] + C[-4, I]) / 2.0
        C = self.ghosts(C)
        C[:, I, 0] = (4.0 * C[:, I, 1] - C[:, I, 2]) / 3.0
        C[:, I, -1] = (5.0 * C[:, I, -2] - 4.0 * C[:, I, -3] + C[:, I, -4]) / 2.0
        P = self.inside(P, P[I, I, I] + C[I, I, I])
        g = self.grad(C)
        U = [self.inside(F, F[I, I, I] - dt * g[q]) for q, F in enumerate(U)]
        for q, F in enumerate(U):
            F[0, I] = 0.0 if c is None or q < 2 else c
            F[-1, I] = (4.0 * F[-2, I] - F[-3, I]) / 3.0
            F[:, I, -1] = (4.0 * F[:, I, -2] - F[:, I, -3]) / 3.0
        P = P.clone()
        self.pressure_faces(U, P, old)
        U, P = [self.ghosts(F) for F in U], self.ghosts(P)
        self.ran += 1
        return U, P, C

    def pressure_faces(self, U, P, old):
        (u, v, w), m, re, I = U, self.m, self.rp.re, slice(1, -1)
        h1, h2 = self.x3[1] - self.x3[0], self.x3[2] - self.x3[0]
        w0, w1, w2 = w[0, I, I], w[1, I, I], w[2, I, I]
        visc = ((w[0, I, :-2] + w[0, I, 2:] - 2 * w0) / m.dx ** 2 + (w[0, :-2, I] + w[0, 2:, I] - 2 * w0) / m.dy ** 2 +
                2 * (h1 * w2 - h2 * w1 + (h2 - h1) * w0) / (h1 * h2 ** 2 - h2 * h1 ** 2))
        P[0, I, I] = P[1, I, I] - (visc / re - w0 * (w1 - w0) / h1) * h1
        P[-1, I, I] = (11 * w[-1, I, I] - 18 * w[-2, I, I] + 9 * w[-3, I, I] - 2 * w[-4, I, I]) / (6 * m.dxi) * self.jinv[-1] / re
        P[I, I, -1] = (3 * u[I, I, -1] - 4 * u[I, I, -2] + u[I, I, -3]) / (2 * m.dx * re)
        f = u[:, :, 0]
        u0, jk = f[I, I], self.jinv[1:-1, None]
        dz = (f[2:, I] - f[:-2, I]) / (2 * m.dxi)
        zz = (f[2:, I] - 2 * u0 + f[:-2, I]) / m.dxi ** 2
        adv = u0 * (u[I, I, 1] - u0) / m.dx + v[I, I, 0] * (f[I, 2:] - f[I, :-2]) / (2 * m.dy) + w[I, I, 0] * dz * jk
        dz, zz = dz.clone(), zz.clone()
        dz[0], dz[-1] = (f[2, I] - f[1, I]) / m.dxi, (f[-2, I] - f[-3, I]) / m.dxi
        zz[0], zz[-1] = (f[3, I] - 2 * f[2, I] + f[1, I]) / m.dxi ** 2, (f[-4, I] - 2 * f[-3, I] + f[-2, I]) / m.dxi ** 2
        visc = ((u0 + u[I, I, 2] - 2 * u[I, I, 1]) / m.dx ** 2 + (f[I, 2:] + f[I, :-2] - 2 * u0) / m.dy ** 2 +
                zz * jk ** 2 - self.j2[1:-1, None] * dz * jk ** 3)
        P[I, I, 0] = (2 * m.dx * ((u0 - old[I, I]) / self.rp.dt + adv - visc / re) - P[I, I, 2] + 4 * P[I, I, 1]) / 3.0

    def shear(self, U):
        """Patch and span average of (dw/dx + du/dz)/Re at the wall."""
        x, m = self.m.x1, self.m
        lo, hi = (f * self.c["lx"] for f in PATCH)
        h1, h2 = self.x3[1] - self.x3[0], self.x3[2] - self.x3[0]
        u, w = U[0][:, 1:-1], U[2][0, 1:-1]
        du = ((u[2] - u[0]) * h1 ** 2 + (u[0] - u[1]) * h2 ** 2) / (h2 * h1 ** 2 - h2 ** 2 * h1)
        tot = []
        for i in range(1, self.nx - 1):
            if not lo <= x[i] <= hi:
                continue
            if i <= 2 or i >= self.nx - 3:
                dw = (w[:, i + 1] - w[:, i - 1]) / (2 * m.dx)
            else:
                dw = (45 * (w[:, i + 1] - w[:, i - 1]) - 9 * (w[:, i + 2] - w[:, i - 2]) + w[:, i + 3] - w[:, i - 3]) / (60 * m.dx)
            tot.append((dw + du[:, i]) / self.rp.re)
        return torch.stack(tot).mean()


def exact(case, seed):
    mesh, rp, st = _problem(case, seed)
    E = _Exact(case, mesh, rp, st)
    U = [torch.tensor(st[f].T.copy(), device="cuda") for f in ("u", "v", "w")]
    P = torch.tensor(st["p"].T.copy(), device="cuda")
    adj = case["kind"] == "adjoint"
    ir = rp.irec - 1
    plane = lambda U: [F[:, 1:-1, ir] - E.mean[q][:, ir, None] for q, F in enumerate(U)]
    file = [f.clone() for f in plane(U)]
    if case["variant"] == 2:
        file = [torch.zeros_like(f) for f in file]
    c = torch.tensor(_control(case, seed).T.copy(), device="cuda") if adj else None
    start = [*U, P]
    if adj:
        for t in (c, *start):
            t.requires_grad_(True)
    live, J = plane(U), 0.0
    with torch.set_grad_enabled(adj):
        live = plane(U)
        for _ in range(case["steps"]):
            U, P, C = E.step(U, P, live, file, c)
            if adj:
                J = J + E.shear(U) / case["steps"]
            if case["variant"] != 2:
                live = plane(U)
    if adj:
        J.backward()
        g = [t.grad.cpu().numpy().T for t in (c, *start)]
        return dict(J=J.item(), dc=g[0], **{"d" + f: a for f, a in zip(("u", "v", "w", "p"), g[1:])})
    return dict(zip(FIELDS, (t.cpu() for t in (*U, P, C))))
