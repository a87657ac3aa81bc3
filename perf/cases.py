"""Performance cases: what a user has this solver do, at the sizes it is used at.

One pass is a short run through the solver's public calls: a state is handed over
(`set_state`, from pinned host memory), the clock is set as a restart does
(`set_time`), some adaptive steps are taken (`solve`) and the state is read back
(`get_state`).  The solver handle is kept between passes, as a program that runs
one configuration many times keeps it.

`exact` restates the scheme in plain float64 torch: reconstruction, troubled-cell
selection, WENO-AO, limiter, Riemann fluxes, sources and the adaptive Runge-Kutta
step.  The stencil weights are an input of the scheme, fixed by the configuration,
and are taken as given.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kfvm-kokkos_b200"))

import kfvm  # noqa: E402
import kfvm_abi as abi  # noqa: E402

DENS, MOMX, MOMY, MOMZ, ETOT, MAGX, MAGY, MAGZ, PSI = range(9)
EPS = 1e-300


# ---------------------------------------------------------------------------
# the cases

def _case(problem, nx, ny, nz, steps, form="fp64", bc=""):
    return {"problem": problem, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "form": form, "bc": bc}


def listed():
    named = {
        # the smallest grids of tests and tutorials: launches and latency count
        "vortex_2d_32": _case("isentropic_vortex", 32, 32, 1, 4),
        # the vortex accuracy test at its stated size
        "vortex_2d_128": _case("isentropic_vortex", 128, 128, 1, 8),
        # production 2D Euler grid
        "kelvin_helmholtz_2d_1024": _case("kelvin_helmholtz", 1024, 1024, 1, 8),
        # a 2D grid with odd extents
        "kelvin_helmholtz_2d_701x419": _case("kelvin_helmholtz", 701, 419, 1, 8),
        # production 2D GLM-MHD grid
        "orszag_tang_2d_1024": _case("orszag_tang", 1024, 1024, 1, 4),
        # 2D special-relativistic hydrodynamics
        "sr_riemann_2d_512": _case("sr_riemann_2d", 512, 512, 1, 6),
        # the headline problem and the largest grid: 3D Euler blast, outflow
        "sod_3d_256": _case("sod3d", 256, 256, 256, 4),
        # a ragged 3D grid between walls
        "sod_3d_97x75x51_walls": _case("sod3d", 97, 75, 51, 6, bc="reflecting"),
        # 3D Navier-Stokes
        "taylor_green_3d_160": _case("taylor_green", 160, 160, 160, 4),
        # 3D GLM-MHD
        "orszag_tang_3d_96": _case("orszag_tang_3d", 96, 96, 96, 3),
        # turbulence with WENO forced on every cell
        "stir_turb_3d_96": _case("stir_turb", 96, 96, 96, 3),
        # the 3xTF32 tensor-core form of the reconstruction
        "sod_3d_128_tf32x3": _case("sod3d", 128, 128, 128, 4, form="tf32x3"),
    }
    return [dict(c, name=n) for n, c in named.items()]


# problem: (weight, dimension, smallest and largest cell count, cell-steps of a pass)
_RANGES = {
    "isentropic_vortex": (2, 2, 2 ** 10, 2 ** 18, 2 ** 18),
    "kelvin_helmholtz": (3, 2, 2 ** 12, 2 ** 21, 2 ** 23),
    "orszag_tang": (2, 2, 2 ** 12, 2 ** 20, 2 ** 22),
    "sr_riemann_2d": (2, 2, 2 ** 12, 2 ** 18, 2 ** 21),
    "sod3d": (4, 3, 2 ** 14, 2 ** 24, 2 ** 26),
    "taylor_green": (2, 3, 2 ** 14, 2 ** 23, 2 ** 24),
    "orszag_tang_3d": (1, 3, 2 ** 14, 2 ** 20, 2 ** 21),
    "stir_turb": (1, 3, 2 ** 14, 2 ** 20, 2 ** 21),
}


def draw(rng):
    names = list(_RANGES)
    problem = rng.choices(names, [_RANGES[n][0] for n in names])[0]
    _, dim, lo, hi, budget = _RANGES[problem]
    # cells on a logarithmic scale, the extents up to a factor of two apart
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi / 1.5)))
    side = cells ** (1.0 / dim)
    ext = [max(8, round(side * math.exp(rng.uniform(-0.35, 0.35)))) for _ in range(dim)]
    while math.prod(ext) > hi:
        ext = [max(8, int(e * 0.95)) for e in ext]
    if dim == 2:
        ext.append(1)
    steps = max(1, min(8, int(budget / math.prod(ext))))
    form, bc = "fp64", ""
    if problem in ("sod3d", "kelvin_helmholtz", "taylor_green", "orszag_tang") and rng.random() < 0.2:
        form = "tf32x3"
    if problem == "sod3d" and rng.random() < 0.3:
        bc = "reflecting"
    return _case(problem, ext[0], ext[1], ext[2], steps, form, bc)


def _config(case):
    cfg, _ = abi.workload(case["problem"], scale=case["nx"], steps=case["steps"])
    cfg.nx, cfg.ny, cfg.nz = case["nx"], case["ny"], case["nz"]
    if case["bc"] == "reflecting":
        for f in range(6):
            cfg.bc[f] = abi.KFVM_BC_REFLECTING
    return cfg


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _spacing(cfg):
    d = [(cfg.xup - cfg.xlo) / cfg.nx, (cfg.yup - cfg.ylo) / cfg.ny]
    return d + [(cfg.zup - cfg.zlo) / cfg.nz] if cfg.dim == 3 else d


def _initial(case, seed, dev):
    """The state at the start of a pass, [variable][z][y][x]: the benchmark problem of
    that name with its parameters varied by the seed."""
    cfg = _config(case)
    g = torch.Generator().manual_seed(1000003 * (int(seed) % 1000003) + 17)

    def rnd(lo, hi):
        return lo + (hi - lo) * torch.rand((), generator=g, dtype=torch.float64).item()

    def axis(lo, up, n, dim):
        x = lo + (up - lo) * (torch.arange(n, dtype=torch.float64, device=dev) + 0.5) / n
        return x.view([-1 if d == dim else 1 for d in range(3)])

    X = axis(cfg.xlo, cfg.xup, cfg.nx, 2)
    Y = axis(cfg.ylo, cfg.yup, cfg.ny, 1)
    Z = axis(cfg.zlo, cfg.zup, cfg.nz, 0) if cfg.dim == 3 else torch.zeros(1, 1, 1, dtype=torch.float64, device=dev)
    shape = (cfg.nz if cfg.dim == 3 else 1, cfg.ny, cfg.nx)
    zero = torch.zeros(shape, dtype=torch.float64, device=dev)
    gam, pi = cfg.gamma, math.pi
    u, v, w = zero, zero, zero
    mag = None
    p = case["problem"]
    if p == "isentropic_vortex":
        beta, x0, y0, uf, vf = rnd(4.5, 5.5), rnd(-1, 1), rnd(-1, 1), rnd(0.8, 1.2), rnd(0.8, 1.2)
        r2 = (X - x0) ** 2 + (Y - y0) ** 2
        f = beta / (2 * pi) * torch.exp(0.5 * (1 - r2))
        u, v = uf - (Y - y0) * f, vf + (X - x0) * f
        rho = (1 - (gam - 1) * beta ** 2 / (8 * gam * pi ** 2) * torch.exp(1 - r2)) ** (1 / (gam - 1))
        pr = rho ** gam
    elif p == "sod3d":
        x0, y0, z0, r = rnd(0.45, 0.55), rnd(0.45, 0.55), rnd(0.45, 0.55), rnd(0.18, 0.24)
        inside = (X - x0) ** 2 + (Y - y0) ** 2 + (Z - z0) ** 2 < r * r
        rho, pr = torch.where(inside, rnd(0.9, 1.1), 0.125) + zero, torch.where(inside, rnd(0.8, 1.2), 0.1) + zero
    elif p == "kelvin_helmholtz":
        y0, amp, ph = rnd(0.45, 0.55), rnd(0.008, 0.012), rnd(0, 2 * pi)
        inside = (Y - y0).abs() < 0.25
        rho, u, pr = torch.where(inside, 2.0, 1.0) + zero, torch.where(inside, 0.5, -0.5) + zero, 2.5 + zero
        # per-cell noise, from a hash of the cell's index
        h = torch.arange(zero.numel(), dtype=torch.float64, device=dev).view(shape)
        h = torch.frac(torch.sin(h * 12.9898 + rnd(0, 100)) * 43758.5453).abs()
        v = amp * torch.sin(4 * pi * X + ph) + 1e-3 * (2 * h - 1)
    elif p == "taylor_green":
        m2 = gam * 0.1 ** 2
        a, x0, y0, z0 = rnd(0.9, 1.1), rnd(0, 2 * pi), rnd(0, 2 * pi), rnd(0, 2 * pi)
        u = a * torch.sin(X - x0) * torch.cos(Y - y0) * torch.cos(Z - z0)
        v = -a * torch.cos(X - x0) * torch.sin(Y - y0) * torch.cos(Z - z0)
        q = a * a * (torch.cos(2 * (X - x0)) + torch.cos(2 * (Y - y0))) * (torch.cos(2 * (Z - z0)) + 2) / 16
        rho, pr = 1 + m2 * q, 1 / m2 + q
    elif p in ("orszag_tang", "orszag_tang_3d"):
        x0, y0, a = rnd(0, 1), rnd(0, 1), rnd(0.9, 1.1)
        sx, sy = 2 * pi * (X - x0), 2 * pi * (Y - y0)
        rho, pr = gam * gam + zero, gam + zero
        u, v = -a * torch.sin(sy) + zero, a * torch.sin(sx) + zero
        if cfg.dim == 3:
            w = 0.2 * torch.sin(2 * pi * Z) + zero
        mag = (-torch.sin(sy) + zero, torch.sin(2 * sx) + zero, zero)
    elif p == "sr_riemann_2d":
        x0, y0, v0 = rnd(-0.1, 0.1), rnd(-0.1, 0.1), rnd(0.97, 0.99)
        e, n = X > x0, Y > y0
        rho = torch.where(e | n, 0.1, 0.5) + zero
        pr = torch.where(e & n, 0.01, 1.0) + zero
        u, v = torch.where(~e & n, v0, 0.0) + zero, torch.where(e & ~n, v0, 0.0) + zero
    else:  # stir_turb: driven turbulence, a sum of long waves at Mach 1
        rho, pr, vel = 1.0 + zero, 1 / gam + zero, []
        for _ in range(3):
            f = zero.clone()
            for _ in range(4):
                k = [int(rnd(0, 4)) for _ in range(3)]
                f += rnd(0.2, 0.4) * torch.sin(2 * pi * (k[0] * X + k[1] * Y + k[2] * Z) + rnd(0, 2 * pi))
            vel.append(f)
        u, v, w = vel
        rho = rho + 0.1 * torch.sin(2 * pi * (X + Y)) + zero
    U = torch.empty((abi.nvars(cfg),) + shape, dtype=torch.float64, device=dev)
    if cfg.eq == abi.KFVM_EQ_SRHYDRO:
        W2 = 1 / (1 - u * u - v * v - w * w)
        m = (rho + gam / (gam - 1) * pr) * W2
        U[DENS], U[ETOT] = rho * W2.sqrt(), m - pr
        U[MOMX], U[MOMY], U[MOMZ] = m * u, m * v, m * w
        vmax = 1.0
    else:
        U[DENS], U[MOMX], U[MOMY], U[MOMZ] = rho, rho * u, rho * v, rho * w
        U[ETOT] = pr / (gam - 1) + 0.5 * rho * (u * u + v * v + w * w)
        c2 = gam * pr / rho
        if mag is not None:
            b2 = mag[0] ** 2 + mag[1] ** 2 + mag[2] ** 2
            U[MAGX], U[MAGY], U[MAGZ], U[PSI] = mag[0], mag[1], mag[2], 0.0
            U[ETOT] += 0.5 * b2
            c2 = c2 + b2 / rho
        vmax = (torch.stack([(x.abs() + zero).max() for x in (u, v, w)]).max() + c2.max().sqrt()).item()
    # the run starts at a fifth of the acoustic step
    return U, 0.2 * cfg.cfl * min(_spacing(cfg)) / vmax


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())


def prepare(case, seed):
    cfg = _config(case)
    U, dt = _initial(case, seed, _device())
    host = _pinned((abi.nvars(cfg), abi.ncells(cfg)))
    host.copy_(U.view(host.shape))
    solver = kfvm.Solver(cfg)
    if case["form"] == "tf32x3":
        solver.set_precision(abi.KFVM_PREC_TF32X3)
    return {"solver": solver, "steps": case["steps"], "dt": dt, "host": host, "in": host.numpy(),
            "out": _pinned(host.shape).numpy()}


def run(state):
    s = state["solver"]
    s.set_state(state["in"])
    s.set_time(0.0, state["dt"])
    s.solve(state["steps"] + 1)  # the step counter starts at 1
    time, _ = s.time_dt()
    return {"state": s.get_state(state["out"]), "time": time}


def work(case):
    """The state in and out once; per cell and evaluation one product per stencil cell,
    direction and variable, the face points' Riemann solves and the update."""
    cfg = _config(case)
    n, nv, d = abi.ncells(cfg), abi.nvars(cfg), cfg.dim
    stencil, points = (13, 2) if d == 2 else (33, 4)
    evals = 4 * case["steps"] + 1
    return {"bytes": 2.0 * n * nv * 8, "flops": float(evals * n * (2 * stencil * d * nv + d * points * 200 + 300))}


def tolerance(case):
    # Differences of rounding (FP64 1e-16, the 3xTF32 sums 1e-7 of the local variation)
    # travel through several adaptive steps and the few decisions at a threshold.
    if case["form"] == "tf32x3":
        return {"rel": 1e-6, "max": 1e-3}
    # The relativistic limiter compares with bounds that hold the cell's own value, so in
    # uniform gas the last rounding decides its theta, and theta < 1 asks for WENO.
    if case["problem"] == "sr_riemann_2d":
        return {"rel": 1e-3, "max": 0.5}
    return {"rel": 1e-9, "max": 1e-6}


# ---------------------------------------------------------------------------
# the scheme in plain float64 torch

def exact(case, seed):
    cfg = _config(case)
    if cfg.eq == abi.KFVM_EQ_SRHYDRO:
        return None  # see tolerance(): rounding decides the cells that use WENO
    U, dt = _initial(case, seed, _device())
    scheme = _Scheme(cfg, U.device)
    U, t = scheme.solve(U, dt, case["steps"])
    return {"state": U.reshape(U.shape[0], -1), "time": t}


def _sq3(a):
    return a[0] * a[0] + a[1] * a[1] + a[2] * a[2]


class _Scheme:
    def __init__(self, cfg, dev):
        self.cfg, self.dev, self.dim, self.eq = cfg, dev, cfg.dim, cfg.eq
        self.nv, self.gam = abi.nvars(cfg), cfg.gamma
        self.glm, self.sr = cfg.eq == abi.KFVM_EQ_MHD_GLM, cfg.eq == abi.KFVM_EQ_SRHYDRO
        self.h = _spacing(cfg)
        self.ext = [cfg.nx, cfg.ny, cfg.nz if self.dim == 3 else 1]
        st = kfvm.stencil(cfg)

        def arr(a, n):
            return torch.tensor(np.array(a)[:, :n] if n else np.array(a), device=dev)

        C, nqf, nqc = st.n_cells, st.nqf, st.nqc
        self.nqf, self.nqc = nqf, nqc
        self.off = np.array(st.off)[:, :C].T.tolist()
        fw = np.array(st.face_w)[: st.n_sub, : 2 * self.dim, :nqf, :C].reshape(st.n_sub, -1, C)
        cw = np.array(st.cell_w)[: st.n_sub, :nqc, :C]
        rows = torch.tensor(np.concatenate([fw, cw], 1) if self.glm else fw, device=dev)
        dw = torch.tensor(np.array(st.deriv_w)[: st.n_sub, : st.n_indic, :C], device=dev)
        # stencil cells of each substencil: the full one, the centre, the biased ones
        sub = [list(range(C)), list(range(st.n_cells_ctr))]
        sub += [list(st.sub_idx[b][: st.n_cells_bias]) for b in range(st.n_bias)]
        self.sub = [torch.tensor(s, device=dev) for s in sub]
        self.rows = [rows[s, :, : len(sub[s])] for s in range(st.n_sub)]
        self.deriv = [dw[s, :, : len(sub[s])] for s in range(st.n_sub)]
        lin = [0.7, 0.3 * 0.7] + [0.3 * (1.0 - 0.7) / st.n_bias] * st.n_bias
        self.lin = torch.tensor(lin, dtype=torch.float64, device=dev)
        # boundary types and the signs that a reflecting wall flips
        self.bc = [cfg.bc[f] for f in range(2 * self.dim)]
        self.sign = []
        for f in range(2 * self.dim):
            s = torch.ones(self.nv, 1, 1, 1, dtype=torch.float64, device=dev)
            if self.bc[f] == abi.KFVM_BC_REFLECTING:
                s[MOMX + f // 2] = -1
                if self.glm:
                    s[MAGX + f // 2] = -1
            self.sign.append(s)

    # ---- equation of state
    def eint(self, U):
        e = U[ETOT] - 0.5 * _sq3(U[MOMX:MOMZ + 1]) / U[DENS]
        return e - 0.5 * _sq3(U[MAGX:MAGZ + 1]) - 0.5 * U[PSI] ** 2 if self.glm else e

    def fast(self, U, b, p):
        a2, b2 = self.gam * p / U[DENS], _sq3(U[MAGX:MAGZ + 1]) / U[DENS]
        s = a2 + b2
        return (0.5 * (s + (s * s - 4 * a2 * b * b / U[DENS]).clamp_min(0).sqrt())).sqrt()

    def prim(self, U):
        """rho, velocities, pressure (SR: and the Lorentz factor)"""
        if not self.sr:
            return [U[DENS], U[MOMX] / U[DENS], U[MOMY] / U[DENS], U[MOMZ] / U[DENS], (self.gam - 1) * self.eint(U)]
        D, E, S2, gm = U[DENS], U[ETOT], _sq3(U[MOMX:MOMZ + 1]), self.gam - 1
        d = E * E - S2
        b = (self.gam - 2) * E
        p = 0.5 * (b + (b * b - 4 * gm * (D * d.sqrt() - d)).clamp_min(0).sqrt())
        p = torch.where(D >= d / E, torch.zeros_like(p), p)
        for _ in range(30):  # Newton's iteration on the pressure
            EP = E + p
            rt = (EP * EP - S2).sqrt()
            p = p + -(S2 + EP * (p / gm - E) + D * rt) / ((2 * p - (self.gam - 2) * E) / gm + D * EP / rt)
        W = 1 / (1 - S2 / (E + p) ** 2).sqrt()
        m = E + p
        return [D / W, U[MOMX] / m, U[MOMY] / m, U[MOMZ] / m, p, W]

    def indicator(self, U):
        return U[DENS] if self.sr else (self.gam - 1) * self.eint(U) / U[DENS] ** self.gam

    def ediff(self, U):
        return U[ETOT] - (U[DENS] ** 2 + _sq3(U[MOMX:MOMZ + 1])).sqrt()

    # ---- halo and stencil access
    def pad(self, U):
        for d in range(self.dim):
            ax, n = 3 - d, self.ext[d]
            per = self.bc[2 * d] == abi.KFVM_BC_PERIODIC
            lo = U.narrow(ax, n - 2, 2) if per else U.narrow(ax, 0, 2).flip(ax) * self.sign[2 * d]
            hi = U.narrow(ax, 0, 2) if per else U.narrow(ax, n - 2, 2).flip(ax) * self.sign[2 * d + 1]
            U = torch.cat([lo, U, hi], ax)
        return U

    def at(self, P, o):
        z = P.narrow(1, 2 + o[2], self.ext[2]) if self.dim == 3 else P
        return z.narrow(2, 2 + o[1], self.ext[1]).narrow(3, 2 + o[0], self.ext[0])

    def ring(self):
        r = range(-1, 2)
        return [(x, y, z) for x in r for y in r for z in (r if self.dim == 3 else (0,))]

    # ---- WENO-AO of listed cells
    def weno(self, P, cells, R):
        nx, ny, nz = self.ext
        py, px = P.shape[2], P.shape[3]
        hz = 2 if self.dim == 3 else 0
        flat, out = P.reshape(self.nv, -1), R.view(R.shape[0], self.nv, -1)
        rel = torch.tensor([(o[2] * py + o[1]) * px + o[0] for o in self.off], device=self.dev)
        for c in cells.split(1 << 16):
            k, j, i = c // (nx * ny), c // nx % ny, c % nx
            base = ((k + hz) * py + j + 2) * px + i + 2
            S = flat[:, base[:, None] + rel]  # [v][cell][stencil cell]
            ref = flat[:, base][:, :, None]
            rho, m = ref[DENS], ref[MOMX:MOMZ + 1]
            V = S.clone()
            if self.sr:
                V[MOMX:MOMZ + 1] = S[MOMX:MOMZ + 1] / rho - S[DENS] * m / rho ** 2
            else:
                u = m / rho
                q = 0.5 * _sq3(u)
                V[MOMX:MOMZ + 1] = (S[MOMX:MOMZ + 1] - u * S[DENS]) / rho
                e = q * S[DENS] + S[ETOT] - (u * S[MOMX:MOMZ + 1]).sum(0)
                if self.glm:
                    e = e - (ref[MAGX:PSI + 1] * S[MAGX:PSI + 1]).sum(0)
                V[ETOT] = (self.gam - 1) * e
            om = torch.stack([(V[:, :, s] @ d.T).square().sum(2) for s, d in zip(self.sub, self.deriv)])
            om = self.lin.view(-1, 1, 1) / (om * om + 1e-40)
            om = om / om.sum(0)
            top = om[0] / self.lin[0]
            om = torch.cat([top[None], om[1:] - top * self.lin[1:].view(-1, 1, 1)])
            r = sum(om[n][:, :, None] * (V[:, :, s] @ w.T) for n, (s, w) in enumerate(zip(self.sub, self.rows)))
            if self.sr:
                r[MOMX:MOMZ + 1] = r[DENS] * m / rho + rho * r[MOMX:MOMZ + 1]
            else:
                e = q * r[DENS] + (rho * u * r[MOMX:MOMZ + 1]).sum(0) + r[ETOT] / (self.gam - 1)
                if self.glm:
                    e = e + (ref[MAGX:PSI + 1] * r[MAGX:PSI + 1]).sum(0)
                r[ETOT] = e
                r[MOMX:MOMZ + 1] = rho * r[MOMX:MOMZ + 1] + u * r[DENS]
            out[:, :, c] = r.permute(2, 0, 1)

    # ---- positivity limiter
    def limit(self, P, R):
        ref = self.at(P, (0, 0, 0))
        near = [self.at(P, o) for o in self.ring()]
        big = torch.full_like(ref[0], 1.7976931348623157e308)
        hi, lo, ei, snd = -big, big, big, big
        for s in near:
            hi, lo = torch.fmax(hi, s[DENS]), torch.fmin(lo, s[DENS])
            if self.sr:
                ei = torch.fmin(ei, self.ediff(s))
            else:
                e = self.eint(s)
                ei = torch.fmin(ei, e)
                snd = torch.fmin(snd, (self.gam * (self.gam - 1) * e / s[DENS]).sqrt())
        if not self.sr:
            div = torch.zeros_like(hi)
            for d in range(self.dim):
                o = [0, 0, 0]
                o[d] = 1
                a, b = self.at(P, o), self.at(P, [-x for x in o])
                div += (a[MOMX + d] / a[DENS] - b[MOMX + d] / b[DENS]) / 2
            eta = torch.fmax(torch.zeros_like(snd), -(0.2 * snd + div) / (0.2 * snd)).clamp_max(1)
            kap = 0.2 * (1 - eta)
            hi, lo, ei = hi * (1 + kap), lo * (1 - kap), ei * (1 - kap)
        one, r0 = torch.ones_like(hi), ref[DENS]
        th = one
        for r in R:
            x = r[DENS]
            low, high = (x < lo, x > hi) if self.sr else (~(x > lo), ~(x < hi))
            th = torch.where(low, torch.fmin(th, (r0 - lo) / (r0 - x)), th)
            th = torch.where(high, torch.fmin(th, (hi - r0) / (x - r0)), th)
        self.mix(R, ref, th)
        th2 = one
        for r in R:
            if self.sr:
                e, e0 = self.ediff(r), self.ediff(ref)
                th2 = torch.where(e < ei, torch.fmin(th2, (e0 - ei) / (e0 - e)), th2)
                continue
            bad = (~(self.eint(r) > ei)).flatten().nonzero().squeeze(1)
            if bad.numel():
                s, c = r.reshape(self.nv, -1)[:, bad], ref.reshape(self.nv, -1)[:, bad]
                m = ei.flatten()[bad]
                a, b = torch.zeros_like(m), torch.ones_like(m)
                for _ in range(10):
                    mid = 0.5 * (a + b)
                    ok = self.eint(c + mid * (s - c)) > m
                    a, b = torch.where(ok, mid, a), torch.where(ok, b, mid)
                th2 = th2.flatten().index_put((bad,), torch.fmin(th2.flatten()[bad], a)).view_as(th2)
        self.mix(R, ref, th2)
        return torch.fmin(th, th2)

    def mix(self, R, ref, th):
        c = (th < 1).flatten().nonzero().squeeze(1)
        if c.numel():
            out, m = R.view(R.shape[0], self.nv, -1), ref.reshape(self.nv, -1)[:, c]
            t = th.flatten()[c].clamp_min(0)
            out[:, :, c] = m + t * (out[:, :, c] - m)

    # ---- the two states at the faces of direction d, point q
    def faces(self, R, d, q):
        ax, n = 3 - d, self.ext[d]
        hi, lo = R[(2 * d + 1) * self.nqf + q], R[2 * d * self.nqf + q]
        if self.bc[2 * d] == abi.KFVM_BC_PERIODIC:
            return torch.cat([hi.narrow(ax, n - 1, 1), hi], ax), torch.cat([lo, lo.narrow(ax, 0, 1)], ax)
        return (torch.cat([lo.narrow(ax, 0, 1) * self.sign[2 * d], hi], ax),
                torch.cat([lo, hi.narrow(ax, n - 1, 1) * self.sign[2 * d + 1]], ax))

    def flux(self, U, V, d):
        F = torch.empty_like(U)
        un, p = V[1 + d], V[4]
        n = MOMX + d
        if self.glm:
            b, ch = U[MAGX:MAGZ + 1], self.ch
            bn, ub = b[d], V[1] * b[0] + V[2] * b[1] + V[3] * b[2]
            pt = p + 0.5 * _sq3(b)
            F[DENS] = U[n]
            for k in range(3):
                F[MOMX + k] = U[n] * V[1 + k] - bn * b[k]
                F[MAGX + k] = un * b[k] - V[1 + k] * bn
            F[n] += pt
            F[MAGX + d] = ch * U[PSI]
            F[ETOT] = un * (U[ETOT] + pt - 0.5 * U[PSI] ** 2) + bn * (ch * U[PSI] - ub)
            F[PSI] = ch * bn
            return F
        F[:4] = U[:4] * un
        F[n] += p
        F[ETOT] = U[n] if self.sr else un * (U[ETOT] + p)
        return F

    def speeds(self, L, R, vL, vR, d):
        uL, uR, g = vL[1 + d], vR[1 + d], self.gam
        if self.sr:
            out = []
            for V in (vL, vR):
                h = 1 + g * V[4] / ((g - 1) * V[0])
                a2 = g * V[4] / (V[0] * h)
                s = a2 / (V[5] ** 2 * (1 - a2))
                r = (s * (1 + s - V[1 + d] ** 2)).sqrt()
                out.append(((V[1 + d] - r) / (1 + s), (V[1 + d] + r) / (1 + s)))
            return torch.minimum(out[0][0], out[1][0]), torch.maximum(out[0][1], out[1][1])
        wL, wR = L[DENS].sqrt(), R[DENS].sqrt()
        if self.glm:
            cL, cR = self.fast(L, L[MAGX + d], vL[4]), self.fast(R, R[MAGX + d], vR[4])
            ch = torch.full_like(cL, self.ch)
            sL = torch.minimum(uL - torch.maximum(ch, cL), uR - torch.maximum(ch, cR))
            sR = torch.maximum(uL + torch.maximum(ch, cL), uR + torch.maximum(ch, cR))
            db = _sq3(L[MAGX:MAGZ + 1] - R[MAGX:MAGZ + 1]).sqrt() / (wL + wR)
            um = (wL * uL + wR * uR) / (wL + wR)
            return torch.minimum(sL, torch.minimum(uL, um) - cL - db), torch.maximum(sR, torch.minimum(uR, um) + cR + db)
        roe = [(wL * a + wR * b) / (wL + wR) for a, b in zip(vL[1:4], vR[1:4])]
        H = (wL * (L[ETOT] + vL[4]) / L[DENS] + wR * (R[ETOT] + vR[4]) / R[DENS]) / (wL + wR)
        a = ((g - 1) * (H - 0.5 * _sq3(roe))).sqrt()
        aL, aR = (g * vL[4] / L[DENS]).sqrt(), (g * vR[4] / R[DENS]).sqrt()
        return torch.minimum(uL - aL, roe[d] - a), torch.maximum(uR + aR, roe[d] + a)

    def riemann(self, L, R, d):
        vL, vR = self.prim(L), self.prim(R)
        sL, sR = self.speeds(L, R, vL, vR, d)
        top = torch.maximum(sL.abs(), sR.abs())
        FL, FR = self.flux(L, vL, d), self.flux(R, vR, d)
        if self.cfg.rs != abi.KFVM_RS_HLLC:
            if self.cfg.rs == abi.KFVM_RS_LLF:
                sL, sR = -top, top
            tR = (sR.clamp_max(0) - sL.clamp_max(0)) / (sR - sL)
            tD = 0.5 * (sR * sL.abs() - sL * sR.abs()) / (sR - sL)
            return (1 - tR) * FL + tR * FR - tD * (R - L), top.max()
        # HLLC with the low-Mach pressure and shear corrections
        g, n, uL, uR, pL, pR = self.gam, MOMX + d, vL[1 + d], vR[1 + d], vL[4], vR[4]
        M = torch.maximum(_sq3(vL[1:4]) * L[DENS] / (g * pL), _sq3(vR[1:4]) * R[DENS] / (g * pR)).sqrt()
        qL, qR = L[DENS] * (sL - uL), R[DENS] * (sR - uR)
        sS = (pR - pL + qL * uL - qR * uR) / (qL - qR)
        pS = 0.5 * (pL + pR + qL * (sS - uL) + qR * (sS - uR))
        psi = -qR * qL / (qL - qR)
        ratio = (torch.minimum(pL, pR) / torch.maximum(pL, pR)).clamp_max(1)
        shear = psi * -torch.expm1(M * ratio.log())
        M = M.clamp_max(1)
        low = psi * (M * (4 + (1 - M * M) ** 2).sqrt() / (1 + M * M) - 1) * (uR - uL)

        def star(U, F, s):
            f = sS / (s - sS) * (s * U - F)
            pf = low + s * pS / (s - sS)
            for k in range(3):
                f[MOMX + k] += pf if k == d else shear * s / (s - sS) * (vR[1 + k] - vL[1 + k])
            f[ETOT] += sS * pf
            return f

        F = torch.where(sR > 0, star(R, FR, sR), FR)
        F = torch.where(sS >= 0, star(L, FL, sL), F)
        return torch.where(sL >= 0, FL, F), top.max()

    # ---- one evaluation of the right-hand side
    def rhs(self, U):
        cfg, cells = self.cfg, U[0].numel()
        P = self.pad(U)
        sparse = self.sparse
        if not sparse:
            self.sparse = cfg.weno_thresh > 0
        nr = self.rows[0].shape[0]
        R = torch.zeros((nr,) + tuple(U.shape), dtype=torch.float64, device=self.dev)
        if sparse:
            for c, o in enumerate(self.off):
                s = self.at(P, o)
                for r in range(nr):
                    R[r].add_(s, alpha=self.rows[0][r, c].item())
            jump = torch.zeros_like(U[0])
            for d in range(self.dim):
                n, ax = self.ext[d], 2 - d
                for q in range(self.nqf):
                    a, b = self.faces(R, d, q)
                    j = (self.indicator(a) - self.indicator(b)).abs()
                    jump = torch.fmax(jump, torch.fmax(j.narrow(ax, 0, n), j.narrow(ax, 1, n)))
            flag = (self.theta < 1) | (jump / self.indicator(U) >= cfg.weno_thresh * min(self.h) ** 1.5)
            if flag.any():
                self.wset = flag
            listed = self.wset.flatten().nonzero().squeeze(1)
        else:
            listed = torch.arange(cells, device=self.dev)
        self.weno(P, listed, R)
        self.theta = self.limit(P, R)
        if self.glm:
            lam = vel = torch.zeros((), dtype=torch.float64, device=self.dev)
            for r in R[: 2 * self.dim * self.nqf]:
                v = (r[MOMX] / r[DENS]).abs()
                lam = torch.maximum(lam, (self.fast(r, r[MAGX], (self.gam - 1) * self.eint(r)) + v).max())
                vel = torch.maximum(vel, v.max())
            self.ch = (lam - vel).item()
        K = torch.zeros_like(U)
        for d in range(self.dim):
            n, ax = self.ext[d], 3 - d
            for q in range(self.nqf):
                F, top = self.riemann(*self.faces(R, d, q), d)
                self.top = max(self.top, top.item())
                K += (F.narrow(ax, 0, n) - F.narrow(ax, 1, n)) / (self.nqf * self.h[d])
        if self.glm:
            self.glm_sources(U, P, R, K)
        if cfg.eq == abi.KFVM_EQ_NAVIERSTOKES:
            self.viscous(P, K)
        return K

    def glm_sources(self, U, P, R, K):
        d2, nq, nf = self.dim == 2, 2, 2 * self.dim * self.nqf
        D = ((-2.7320508075688767, 1.732050807568877, 1.7320508075688767, -0.7320508075688767),
             (0.7320508075688767, -1.7320508075688767, -1.732050807568877, 2.7320508075688767))
        div = torch.zeros_like(U[0])
        for d in range(self.dim):
            for q in range(self.nqf):
                a, b = self.faces(R, d, q)
                m = 0.5 * (a[MAGX + d] + b[MAGX + d])
                div += (m.narrow(2 - d, 1, self.ext[d]) - m.narrow(2 - d, 0, self.ext[d])) / (self.nqf * self.h[d])
        smooth = self.theta >= 0.75
        pts = [(x, y, z) for x in range(nq) for y in range(nq) for z in range(1 if d2 else nq)]

        def inner(p):
            return R[nf + (p[0] * nq + p[1] if d2 else (p[0] * nq + p[1]) * nq + p[2])]

        for p in pts:
            s = inner(p)
            v = s[MOMX:MOMZ + 1] / s[DENS]
            grad = torch.zeros_like(div)
            for d in range(self.dim):
                o = [0, 0, 0]
                o[d] = 1
                plain = (self.at(P, o)[PSI] - self.at(P, [-x for x in o])[PSI]) / (2 * self.h[d])
                t = [p[k] for k in range(self.dim) if k != d]
                q = t[0] if d2 else t[0] * nq + t[1]
                fine = D[p[d]][0] * R[2 * d * self.nqf + q][PSI] + D[p[d]][3] * R[(2 * d + 1) * self.nqf + q][PSI]
                for m in range(nq):
                    fine = fine + D[p[d]][1 + m] * inner(tuple(m if k == d else p[k] for k in range(3)))[PSI]
                grad += v[d] * torch.where(smooth, fine / self.h[d], plain)
            w, b = 1.0 / len(pts), s[MAGX:MAGZ + 1]
            K[MOMX:MOMZ + 1] -= w * div * b
            K[ETOT] -= w * (div * (v * b).sum(0) + grad * s[PSI])
            K[MAGX:MAGZ + 1] -= w * div * v
            K[PSI] -= w * grad

    def viscous(self, P, K):
        q = {}
        for o in self.ring():
            s = self.at(P, o)
            v = [s[MOMX + k] / s[DENS] for k in range(3)]
            q[o] = v + [(self.gam - 1) * self.eint(s) / s[DENS]]

        def unit(d, n=1):
            return tuple(n if k == d else 0 for k in range(3))

        def add(a, b):
            return tuple(x + y for x, y in zip(a, b))

        def grad_normal(k, a, d):  # between the cells a and a + e_d
            return (q[add(a, unit(d))][k] - q[a][k]) / self.h[d]

        def grad_side(k, a, d, t):  # along t, at the face between a and a + e_d
            # (the scheme averages the x derivatives at z faces over the cell's y neighbour)
            b = add(a, unit(1 if (d, t) == (2, 0) else d))
            return (q[add(a, unit(t))][k] + q[add(b, unit(t))][k] - q[add(a, unit(t, -1))][k]
                    - q[add(b, unit(t, -1))][k]) / (4 * self.h[t])

        S = [torch.zeros_like(K[0]) for _ in range(4)]
        re, pr = self.cfg.reynolds, self.cfg.prandtl
        for d in range(self.dim):
            for a, sgn in (((0, 0, 0), 1.0), (unit(d, -1), -1.0)):
                for k in range(3):
                    if k == d:
                        f = 4.0 / 3.0 * grad_normal(d, a, d)
                        for t in range(self.dim):
                            if t != d:
                                f = f - 2.0 / 3.0 * grad_side(t, a, d, t)
                    else:
                        f = grad_normal(k, a, d)
                        if k < self.dim:
                            f = f + grad_side(d, a, d, k)
                    S[k] += sgn * f / (self.h[d] * re)
                S[3] += sgn * grad_normal(3, a, d) / (self.h[d] * re * pr)
        c = q[(0, 0, 0)]
        for k in range(3):
            K[MOMX + k] += S[k]
        K[ETOT] += S[3] + c[0] * S[0] + c[1] * S[1] + c[2] * S[2]

    # ---- adaptive SSP(4,3) steps with the first-same-as-last stage
    def solve(self, U, dt, steps):
        cfg = self.cfg
        self.theta, self.wset = torch.ones_like(U[0]), torch.zeros_like(U[0], dtype=torch.bool)
        self.sparse, self.top, self.ch = cfg.weno_thresh > 0, 0.0, 0.0
        K, t, err, dmin = self.rhs(U), 0.0, 1.0, min(self.h)
        for _ in range(steps):
            first = True
            for attempt in range(cfg.rejection_limit):
                self.top = 0.0
                if attempt:
                    K = self.rhs(U)
                S, hat = U + 0.5 * dt * K, U + 0.25 * dt * K
                for a, b, c in ((1.0, 0.0, 0.5), (1 / 3, 2 / 3, 1 / 6), (1.0, 0.0, 0.5)):
                    k = self.rhs(S)
                    hat += 0.25 * dt * k
                    S = a * S + c * dt * k
                    if b:
                        S += b * U
                k = self.rhs(S)
                e = ((S - hat) / (cfg.atol + cfg.rtol * torch.maximum(S.abs(), hat.abs()))).square().mean().item()
                new = math.inf if e == 0 else 1 / math.sqrt(e)
                fac = new ** (0.8 / 3) * err ** (-0.31 / 3)
                fac = 1.2 if math.isnan(fac) else 1 + math.atan(fac - 1)
                if self.sr:
                    ok = torch.minimum(S[DENS], S[ETOT] ** 2 - S[DENS] ** 2 - _sq3(S[MOMX:MOMZ + 1])).min() >= 0
                else:
                    ok = torch.minimum(S[DENS], self.eint(S)).min() >= 0
                if not ok:
                    dt = min(0.25 * cfg.cfl * dmin / self.top, dt / 4) if first else dt / 2
                    first, self.sparse = False, False
                elif fac >= cfg.rejection_thresh:
                    U, K, t, err = S, k, t + dt, new
                    dt = min(dt * fac, cfg.cfl * dmin / self.top)
                    break
                else:
                    dt *= fac
            else:
                break  # no attempt was accepted: the run ends
        return U, t
