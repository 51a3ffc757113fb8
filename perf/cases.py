"""The work that a program has this library do, as measurable cases.

Each case is a call pattern of a user's program on one of the named workloads
of disco2_b200.configs:

  run       the main loop between two outputs: n RK2 steps, then the state of
            every disk read back;
  couple    a host code that keeps the state: upload, one step, download;
  survey    n steps, then the reductions of a diagnostics dump (radial
            profiles, equatorial rows, binary torque);
  gradient  an objective run and its reverse sweep, from a given state;
  tangent   the forward-mode derivative along one direction, from a given state.

A case's inputs are the workload's initial state with seeded noise on density
and pressure (the relative amplitude the configurations themselves use for
their noise, at most 1e-3).  Outputs are float64 arrays as the library hands
them out.
"""
from __future__ import annotations

import math

import numpy as np

from disco2_b200 import configs, lib

NOISE = 1.0e-4

# FP64 operations of one cell in one RK2 step (a division, a square root and a
# transcendental count as one), from the formulas: slopes, face list, limiters,
# one phi face and two r faces, sources, update.
FLOPS_STEP = 1400.0
FLOPS_VISC = 500.0   # viscous fluxes of the same faces, viscous heating
FLOPS_Z = 700.0      # two z faces, their slopes and limiter
# Bytes of one cell in one RK2 step: 5 conserved values and 1 phi edge, read
# and written across the two stages (48 + 48, then 96 + 48).
BYTES_STEP = 240.0


def listed():
    return [
        # a host program that owns the state and calls one small step at a time
        {"name": "couple_gresho_24", "do": "couple", "workload": "gresho", "num_r": 24, "steps": 1},
        # a 1-D-like disk (two cells per annulus): every launch is nearly empty;
        # the settings of the Shakura-Sunyaev test, outflow, cooling, sink
        {"name": "sstest_128", "do": "run", "workload": "sstest", "num_r": 128, "steps": 60},
        # MacFadyen-Milosavljevic circumbinary disk, outflow and moving frame
        {"name": "milos_128", "do": "run", "workload": "milos_macfadyen", "num_r": 128, "steps": 60},
        # the inviscid vortex on the rigidly rotating mesh
        {"name": "gresho_96", "do": "run", "workload": "gresho", "num_r": 96, "steps": 40},
        # HLL, constant viscosity, one point mass
        {"name": "kepler_ring_256", "do": "run", "workload": "kepler_ring", "num_r": 256, "steps": 60},
        # the headline disk: binary, alpha viscosity, HLLC, outer damping
        {"name": "circumbinary_400", "do": "run", "workload": "circumbinary", "num_r": 400, "steps": 100},
        # the reference's own 3-D parfile
        {"name": "torus3d_80", "do": "run", "workload": "torus3d", "num_r": 80, "num_z": 80, "steps": 60},
        # a parameter sweep: many uneven disks in one context
        {"name": "sweep_12", "do": "run", "workload": "sweep", "disks": 12, "steps": 80},
        # the cadence of a diagnostics dump on an odd-sized disk
        {"name": "survey_circumbinary_157", "do": "survey", "workload": "circumbinary", "num_r": 157, "steps": 20},
        # sensitivities of the torque: one reverse sweep, and one direction
        {"name": "gradient_192", "do": "gradient", "workload": "circumbinary", "num_r": 192, "steps": 50},
        {"name": "tangent_96", "do": "tangent", "workload": "circumbinary", "num_r": 96, "steps": 40},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# workload -> (smallest, largest num_r) of the draws
RANGES = {
    "gresho": (12, 128), "kepler_ring": (16, 320), "circumbinary": (24, 512), "milos_macfadyen": (24, 160),
    "sstest": (24, 256), "vortex_dye": (40, 96), "shear": (24, 128), "rad_dom": (24, 160), "middle": (24, 160),
    "torus": (16, 120), "torus3d": (16, 96), "sweep": (0, 0),
}


def draw(rng):
    do = rng.choice(["run"] * 6 + ["couple", "survey", "gradient", "tangent"])
    if do in ("gradient", "tangent"):
        w = rng.choice(["circumbinary", "kepler_ring"])
        return {"do": do, "workload": w, "num_r": _log_int(rng, 24, 200), "steps": _log_int(rng, 6, 40),
                "q": 10.0 ** rng.uniform(-2.0, 0.0), "alpha": rng.uniform(0.01, 0.1)}
    names = sorted(RANGES) if do == "run" else [n for n in sorted(RANGES) if n not in ("torus3d", "sweep")]
    w = rng.choice(names)
    c = {"do": do, "workload": w, "steps": 1 if do == "couple" else _log_int(rng, 5, 60)}
    if w == "sweep":
        c["disks"] = _log_int(rng, 2, 11)
        c["sweep_seed"] = rng.randint(1, 10**6)
        c["steps"] = _log_int(rng, 5, 40)
        return c
    lo, hi = RANGES[w]
    c["num_r"] = _log_int(rng, lo, hi)
    if w == "torus3d":
        c["num_z"] = _log_int(rng, 8, 96)
    if w == "circumbinary":
        c["q"], c["alpha"] = 10.0 ** rng.uniform(-2.0, 0.0), rng.uniform(0.01, 0.1)
        c["hor"], c["r_max"] = rng.uniform(0.05, 0.1), rng.uniform(10.0, 30.0)
    return c


def _params(case):
    """The parameter dicts of the case's disks."""
    w = case["workload"]
    if w == "sweep":
        return configs.circumbinary_sweep(case["disks"], seed=case.get("sweep_seed", 3))
    kw = {"num_r": case["num_r"]}
    if w == "torus3d":
        kw["num_z"] = case["num_z"]
    if w == "circumbinary":
        for k in ("q", "alpha", "hor", "r_max"):
            if k in case:
                kw[k] = case[k]
    if w == "vortex_dye":
        return [configs.vortex_test(NUM_N=1, **kw)]
    return [configs.WORKLOADS[w](**kw)]


def _input_state(sim, seed, k):
    """Initial state of disk k with seeded relative noise on density and
    pressure."""
    st = sim.initial_state()
    rng = np.random.default_rng([seed, k])
    st["prim"][:, 0] *= 1.0 + NOISE * rng.uniform(-1.0, 1.0, sim.num_cells)
    st["prim"][:, 1] *= 1.0 + NOISE * rng.uniform(-1.0, 1.0, sim.num_cells)
    return st


def _upload(ctx, states):
    for k, st in enumerate(states):
        ctx.set_state(k, st["prim"], st["tiph"], st["dphi"])
        ctx.set_gravmass(k, st["gm"])
        ctx.set_time(k, 0.0)


def prepare(case, seed):
    sims = [lib.Sim(p) for p in _params(case)]
    ctx = lib.Context(sims, device=0)
    states = [_input_state(s, seed, k) for k, s in enumerate(sims)]
    _upload(ctx, states)
    out = {"case": case, "ctx": ctx, "n": len(sims), "steps": case["steps"]}
    if case["do"] in ("couple", "gradient", "tangent"):
        out["states"] = states
    if case["do"] == "tangent":
        out["dprim"] = states[0]["prim"] * np.random.default_rng([seed, 99]).uniform(-1.0, 1.0, (sims[0].num_cells, 1))
    return out


def _readback(ctx, n):
    disks = [ctx.get_state(k) for k in range(n)]
    return {"disks": disks, "gm": np.stack([ctx.gravmass(k) for k in range(n)]),
            "time": np.array([ctx.time(k) for k in range(n)])}


def run(state):
    ctx, do, steps = state["ctx"], state["case"]["do"], state["steps"]
    if do == "run":
        ctx.step(steps)
        return _readback(ctx, state["n"])
    if do == "couple":
        _upload(ctx, state["states"])
        ctx.step(steps)
        return _readback(ctx, state["n"])
    if do == "survey":
        ctx.step(steps)
        return {**ctx.diagnostics(0), "torque": ctx.torque(0)}
    _upload(ctx, state["states"])
    if do == "gradient":
        return ctx.adjoint(steps, steps // 2, ckpt_every=25, weights=(1.0, 0.5))
    J, dJ = ctx.tangent(steps, steps // 2, dq=0.3, dalpha=0.2, dprim=state["dprim"])
    return {"J": J, "dJ": dJ}


def work(case):
    sims = [lib.Sim(p) for p in _params(case)]
    cells = sum(s.num_cells for s in sims)
    per = FLOPS_STEP + (FLOPS_VISC if sims[0].param("Explicit_Viscosity") > 0 else 0.0)
    per += FLOPS_Z if case["workload"] == "torus3d" else 0.0
    state = 8.0 * sum(s.num_cells * (2 * s.num_q + 2) for s in sims)
    io = {"run": 1.0, "couple": 1.6, "survey": 1.5, "gradient": 1.0, "tangent": 1.0}[case["do"]]
    # forward + reverse: the forward steps, their recomputation, and about two
    # evaluations' worth of reverse arithmetic; a tangent is value + derivative
    k = {"gradient": 4.0, "tangent": 3.0}.get(case["do"], 1.0)
    return {"bytes": k * BYTES_STEP * cells * case["steps"] + io * state, "flops": k * per * cells * case["steps"]}


# ---------------------------------------------------------------------------
# The run and couple cases of the Gresho, Keplerian ring and circumbinary disks
# in plain numpy: the moving-mesh RK2 step written over whole arrays.
# ---------------------------------------------------------------------------
EXACT_CELL_STEPS = 1.6e6
TWO_PI = 2.0 * math.pi
RHO, PPP, URR, UPP, UZZ = range(5)


def exact(case, seed):
    if case["do"] not in ("run", "couple") or case["workload"] not in ("gresho", "kepler_ring", "circumbinary"):
        return None
    par = _params(case)[0]
    sim = lib.Sim(par)
    if sim.num_cells * case["steps"] > EXACT_CELL_STEPS:
        return None
    quiet = lib.Sim({**par, "IC_Noise": 0.0}).initial_state()["prim"]
    disk = _Disk(par, *sim.grid(), _input_state(sim, seed, 0), quiet)
    for _ in range(case["steps"]):
        disk.step()
    gm = np.zeros((2, 6))
    gm[:, 0], gm[:, 1], gm[:, 2], gm[:, 3] = disk.gr, disk.gphi, disk.gm, disk.gom
    return {"disks": [{"prim": disk.prim.T.copy(), "cons": disk.cons.T.copy(), "tiph": disk.tiph, "dphi": disk.dphi}],
            "gm": gm[None], "time": np.array([[disk.t, disk.dt]])}


def _pm(x):
    """x moved by whole turns into [-pi, pi]."""
    return x - TWO_PI * np.round(x / TWO_PI)


class _Disk:
    """A 2-D disk with fixed radial boundaries (one ghost annulus a side)."""

    def __init__(self, par, n_p, rf, st, quiet):
        self.par, self.np_, self.nr = par, n_p.astype(int), len(n_p)
        self.off = np.concatenate([[0], np.cumsum(self.np_)])
        self.a = np.repeat(np.arange(self.nr), self.np_)
        self.rm, self.rp = rf[:-1], rf[1:]
        self.rc = 0.5 * (self.rm + self.rp)
        idx = np.arange(self.off[-1])
        first, last = self.off[:-1][self.a], self.off[1:][self.a] - 1
        self.left = np.where(idx == first, last, idx - 1)
        self.right = np.where(idx == last, first, idx + 1)
        # the layer's faces from the log-stretched z coordinate
        zs = par["ZLogScale"]
        zf = [math.copysign(zs * (math.exp(zs * math.log(1.0 + abs(z) / zs) / zs) - 1.0), z)
              for z in (par["Z_Min"], par["Z_Max"])]
        self.dz = zf[1] - zf[0]
        self.gam = par["Adiabatic_Index"]
        self.nu = par["Explicit_Viscosity"]
        kepler = par["w_analytic_type"] == 1
        self.rom = lambda r: r ** -0.5 if kepler else 0.0 * r
        self.rdrom = lambda r: -1.5 * r ** -1.5 if kepler else 0.0 * r
        self.target = quiet[self.off[:-1]].T  # the axisymmetric profile of each annulus
        self.prim, self.tiph, self.dphi = st["prim"].T.copy(), st["tiph"].copy(), st["dphi"].copy()
        self.gr, self.gphi, self.gm, self.gom = (st["gm"][:, k].copy() for k in range(4))
        self.t, self.dt = 0.0, 0.0
        self.cons = self._cons(self.prim)

    def _dv(self):
        return 0.5 * (self.rp ** 2 - self.rm ** 2)[self.a] * self.dphi * self.dz

    def _u(self, p, r):
        """Conserved densities of prims p at radius r."""
        vp = p[UPP] * r
        e = 0.5 * p[RHO] * (p[URR] ** 2 + vp ** 2 + p[UZZ] ** 2) + p[PPP] / (self.gam - 1.0)
        return np.stack([p[RHO], e, p[RHO] * p[URR], r * p[RHO] * vp, p[RHO] * p[UZZ]])

    def _cons(self, p):
        return self._u(p, self.rc[self.a]) * self._dv()

    def _flux(self, p, r, n, u):
        vp = p[UPP] * r
        vn = p[URR] if n == 0 else vp
        f = u * vn
        f[1] += p[PPP] * vn
        f[2 if n == 0 else 3] += p[PPP] * (1.0 if n == 0 else r)
        return f, vn

    def _riemann(self, pl, pr, r, n, w):
        ul, ur = self._u(pl, r), self._u(pr, r)
        fl, vl = self._flux(pl, r, n, ul)
        fr, vr = self._flux(pr, r, n, ur)
        cl, cr = np.sqrt(self.gam * pl[PPP] / pl[RHO]), np.sqrt(self.gam * pr[PPP] / pr[RHO])
        sl, sr = np.minimum(vl - cl, vr - cr), np.maximum(vl + cl, vr + cr)
        ss = (pr[RHO] * vr * (sr - vr) - pl[RHO] * vl * (sl - vl) + pl[PPP] - pr[PPP]) / (
            pr[RHO] * (sr - vr) - pl[RHO] * (sl - vl))
        if self.par["RiemannSolver"] == 1:
            us = (sr * ur - sl * ul + fl - fr) / (sr - sl)
            fs = (sr * fl - sl * fr - sr * sl * (ul - ur)) / (sr - sl)
            star = fs - w * us
        else:
            left = w < ss
            p, u, f, s = np.where(left, pl, pr), np.where(left, ul, ur), np.where(left, fl, fr), np.where(left, sl, sr)
            vn = np.where(left, vl, vr)
            us = (s - vn) / (s - ss) * u
            us[2 if n == 0 else 3] = us[0] * ss * (1.0 if n == 0 else r)
            ps = p[RHO] * (s - vn) * (ss - vn) + p[PPP]
            us[1] = ((s - vn) * u[1] + ps * ss - p[PPP] * vn) / (s - ss)
            star = f + s * (us - u) - w * us
        return np.where(w < sl, fl - w * ul, np.where(w > sr, fr - w * ur, star))

    def _nu(self, p, rho, r, phi, gr, gphi, gm):
        if self.par["ViscConst"] == 1:
            return self.nu
        om2 = 0.0
        for k in range(2):
            d2 = (r * np.cos(phi) - gr[k] * math.cos(gphi[k])) ** 2 + (r * np.sin(phi) - gr[k] * math.sin(gphi[k])) ** 2
            om2 = om2 + gm[k] * (d2 + self.par["G_EPS"] ** 2) ** -1.5
        return self.nu * p / rho / np.sqrt(om2)

    def _faces(self, tiph):
        """Inner cell, outer cell, width, centre and pair of every r face."""
        out = []
        for i in range(self.nr - 1):
            ci, co = slice(self.off[i], self.off[i + 1]), slice(self.off[i + 1], self.off[i + 2])
            p0 = tiph[self.off[i + 1] - 1]
            x = np.mod(tiph[ci] - p0, TWO_PI)
            x[-1] = TWO_PI
            y = np.mod(tiph[co] - p0, TWO_PI)
            k0 = int(np.argmin(y))
            y = np.roll(y, -k0)
            e = np.sort(np.concatenate([x, y]))
            lo = np.concatenate([[0.0], e[:-1]])
            mid = 0.5 * (lo + e)
            j = np.searchsorted(x, mid)
            k = (np.searchsorted(y, mid) + k0) % self.np_[i + 1]
            out.append((self.off[i] + j, self.off[i + 1] + k, e - lo, p0 + mid, np.full(len(e), i)))
        return [np.concatenate(v) for v in zip(*out)]

    def step(self):
        p = self.par
        rk = (self.cons.copy(), self.tiph.copy(), self.gphi.copy(), self.gr.copy(), self.gom.copy())
        for sub, b, fac in ((1, 0.0, 1.0), (2, 0.5, 0.5)):
            self._substep(sub, b, fac, rk)
            # the binary
            turn = np.round((self.gphi - rk[2]) / TWO_PI) * TWO_PI
            self.gphi = (1 - b) * self.gphi + b * (rk[2] + turn)
            m = self.gm.sum()
            om = m ** 1.5  # unit separation; 0 without a mass
            self.gr = self.gm[::-1] / m if m > 1e-12 else np.zeros(2)
            self.gphi = self.gphi + om * fac * self.dt
            self.gom = np.full(2, om)
        self.t += self.dt

    def _substep(self, sub, b, fac, rk):
        par, a, N = self.par, self.a, len(self.a)
        prim, dphi = self.prim, self.dphi
        tw = np.mod(self.tiph, TWO_PI)
        self.gphi = np.mod(self.gphi, TWO_PI)
        r, rm, rp = self.rc[a], self.rm[a], self.rp[a]
        plm = par["PLM"]
        # phi slopes
        dl, dr = 0.5 * (dphi + dphi[self.left]), 0.5 * (dphi + dphi[self.right])
        sl, sr = (prim - prim[:, self.left]) / dl, (prim[:, self.right] - prim) / dr
        sm = (prim[:, self.right] - prim[:, self.left]) / (dl + dr)
        gp = np.sign(sl) * np.minimum(np.minimum(plm * abs(sl), plm * abs(sr)), abs(sm)) * (sl * sr > 0)
        # mesh velocity
        w = np.zeros(self.nr)
        if par["w_numeric_type"] == 2:
            w = np.add.reduceat(r * prim[UPP] * self.cons[0], self.off[:-1]) / np.add.reduceat(self.cons[0], self.off[:-1])
        wa = w[a]
        # r faces and slopes
        cl, cr, fd, cm, pair = self._faces(self.tiph)
        fr_, fdl, fdr = self.rp[pair], 0.5 * (self.rp - self.rm)[pair], 0.5 * (self.rp - self.rm)[pair + 1]
        phi = tw - 0.5 * dphi
        opl, opr = _pm(cm - phi[cl]), _pm(phi[cr] - cm)
        wl, wr = prim[:, cl] + opl * gp[:, cl], prim[:, cr] - opr * gp[:, cr]
        s = (wr - wl) / (fdr + fdl)
        da = fr_ * fd * self.dz
        tot = self.dz * dphi * np.where(a == 0, rp, np.where(a == self.nr - 1, rm, rm + rp))
        g = np.stack([np.bincount(cl, s[q] * da, N) + np.bincount(cr, s[q] * da, N) for q in range(5)]) / tot
        both, ss = np.concatenate([cl, cr]), np.concatenate([s, s], axis=1)
        for q in range(5):
            least, opp = np.full(N, np.inf), np.zeros(N, bool)
            np.minimum.at(least, both, abs(ss[q]))
            np.logical_or.at(opp, both, ss[q] * g[q][both] < 0)
            g[q] = np.where(opp, 0.0, np.sign(g[q]) * np.minimum(abs(g[q]), plm * least))
        # time step
        if sub == 1:
            width = np.minimum(np.minimum(rp - rm, r * dphi), self.dz)
            v = np.sqrt(self.gam * prim[PPP] / prim[RHO]) + np.sqrt(
                prim[URR] ** 2 + (prim[UPP] * r - wa) ** 2 + prim[UZZ] ** 2)
            dt = par["CFL"] * width / v
            if self.nu > 0:
                nu = self._nu(prim[PPP], prim[RHO], r, self.tiph - 0.5 * dphi, rk[3], rk[2], self.gm)
                dt = dt / (1.0 + dt / (0.25 * width ** 2 / nu))
            self.dt = dt[(a > 0) & (a < self.nr - 1)].min()
        dt = fac * self.dt
        cons = (1 - b) * self.cons + b * rk[0]
        # phi faces (j, j+1) at cell j
        R = self.right
        f = self._riemann(prim + 0.5 * gp * dphi, prim[:, R] - 0.5 * gp[:, R] * dphi[R], r, 1, wa)
        if self.nu > 0:
            avg = 0.5 * (prim + prim[:, R])
            width = tw[R] - tw  # wrapped edges: the code's convention at phi = 0
            gph, grr = (prim[:, R] - prim) / width / r, 0.5 * (g + g[:, R])
            x = self._nu(avg[PPP], avg[RHO], r, tw, self.gr, self.gphi, self.gm) * avg[RHO]
            rd = self.rdrom(r)
            srp = r * (r * grr[UPP] + rd) + r * gph[URR]
            f[2] -= x * srp / r
            f[3] -= x * (-r * grr[URR] + avg[URR] + r * r * gph[UPP])
            f[1] -= x * (-r * avg[UPP] * (grr[URR] - avg[URR] / r - r * gph[UPP]) + avg[URR] * (
                gph[URR] + rd + r * grr[UPP]))
        f *= dt * (rp - rm) * self.dz
        cons += f[:, self.left] - f
        # r faces
        f = self._riemann(prim[:, cl] + g[:, cl] * fdl + gp[:, cl] * opl, prim[:, cr] - g[:, cr] * fdr - gp[:, cr] * opr,
                          fr_, 0, 0.0)
        vl = np.zeros_like(f)
        vr = vl
        if self.nu > 0:
            avg, gph = 0.5 * (wl + wr), 0.5 * (gp[:, cl] + gp[:, cr]) / fr_
            x = self._nu(avg[PPP], avg[RHO], fr_, cm, self.gr, self.gphi, self.gm) * avg[RHO]
            rd = self.rdrom(fr_)
            vl = np.zeros_like(f)
            vl[2] = -x * (fr_ * s[URR] - avg[URR] - fr_ * fr_ * gph[UPP])
            vl[3] = -x * (fr_ * (fr_ * s[UPP] + rd) + fr_ * gph[URR])
            vl[1] = -x * (avg[URR] * (s[URR] - avg[URR] / fr_ - fr_ * gph[UPP]) + fr_ * avg[UPP] * (
                gph[URR] + rd + fr_ * s[UPP]))
            vr = vl.copy()
            vl[2] /= fr_ - fdl
            vr[2] /= fr_ + fdr
        for q in range(5):
            cons[q] += np.bincount(cr, (f[q] + vr[q]) * dt * da, N) - np.bincount(cl, (f[q] + vl[q]) * dt * da, N)
        # sources
        dv = self._dv()
        c_, s_ = np.cos(phi), np.sin(phi)
        fr, fp = np.zeros(N), np.zeros(N)
        n, eps = par["PHI_ORDER"], par["G_EPS"]
        for k in range(2):
            dx = r * c_ - self.gr[k] * math.cos(self.gphi[k])
            dy = r * s_ - self.gr[k] * math.sin(self.gphi[k])
            d = np.hypot(dx, dy)
            f1 = -self.gm[k] * d ** (n - 1.0) / (d ** n + eps ** n) ** (1.0 + 1.0 / n)
            fr += f1 * (dx * c_ + dy * s_) / d
            fp += f1 * (dy * c_ - dx * s_) / d
        rho, vp, vr_ = prim[RHO], prim[UPP] * r, prim[URR]
        om, rd = self.rom(r), self.rdrom(r)
        fc = om * om / r
        cons[2] += dt * dv * ((rho * vp * vp + prim[PPP]) / r + rho * (fr + fc))
        cons[3] += dt * dv * rho * fp * r
        cons[1] += dt * dv * rho * ((fr + fc) * vr_ + (fp - vr_ * rd) * vp)
        if self.nu > 0:
            x = rho * self._nu(prim[PPP], rho, r, phi, self.gr, self.gphi, self.gm)
            cons[1] += dt * dv * x * rd * (rd + r * g[UPP] + gp[URR])
        # epicyclic rotation
        big, slope = om / r, 2.0 * om + r * rd
        k2 = 2.0 * big / r * slope
        kap = np.sqrt(np.where(k2 > 0, k2, 1.0))
        ck, sk = np.cos(kap * dt), np.sin(kap * dt)
        l0, r0 = cons[3].copy(), cons[2].copy()
        cons[3] = np.where(k2 > 0, l0 * ck - r0 * slope / kap * sk, l0)
        cons[2] = np.where(k2 > 0, r0 * ck + 2.0 * big * l0 / r / kap * sk, r0)
        # mesh motion
        old = rk[1] + np.round((tw - rk[1]) / TWO_PI) * TWO_PI
        self.tiph = (1 - b) * tw + b * old + (wa + om) * dt / r
        self.dphi = np.mod(self.tiph - self.tiph[self.left], TWO_PI)
        # prims, boundary, damping
        u = cons / self._dv()
        rho = np.maximum(u[0], par["Rho_Floor"])
        v = np.stack([u[2], u[3] / r, u[4]]) / rho
        ke = 0.5 * rho * (v * v).sum(0)
        pp = (self.gam - 1.0) * (u[1] - ke)
        pp = np.clip(pp, par["Cs_Floor"] ** 2 * rho / self.gam, par["Cs_Cap"] ** 2 * rho / self.gam)
        mag = np.sqrt((v * v).sum(0))
        v *= np.where(mag > par["Vel_Cap"], par["Vel_Cap"] / np.maximum(mag, 1e-300), 1.0)
        prim = np.stack([rho, pp, v[0], v[1] / r, v[2]])
        ghost = (a == 0) | (a == self.nr - 1)
        prim = np.where(ghost, self.target[:, a], prim)
        if par["DAMP_TIME"] > 0:
            rate = (r - par["RDAMP_OUTER"]) / (par["R_Max"] - par["RDAMP_OUTER"]) / par["DAMP_TIME"] / TWO_PI
            prim = prim + np.where(r > par["RDAMP_OUTER"], -np.expm1(-rate * dt), 0.0) * (self.target[:, a] - prim)
        self.prim = prim
        self.cons = self._cons(prim)
