"""Performance cases: what a user of nebulasem_gb300 has it compute, over the
range of its workloads, through the public Solver calls.

Every case is a rising thermal bubble in a box of nx x ny x nz hexahedral
elements of edge h and order N (2D: one element thick in y), as the package's
workloads and tests build it, with a smooth wind of up to about 1 m/s so that
no term of the equations is at rest.  The state comes from pinned host arrays
and goes back to them, as a host code that owns the fields does.

  kind        one pass
  tendency    state in, one right-hand side in the precision form, back
  step        state in, `steps` SSP-RK3 steps (prec: fp64 or mixed), state out
  segregated  fields in, `steps` steps of the reference's own update, fields out
  convection  wind and scalar in, `steps` convection steps, scalar out
  adjoint     state in, checkpointed forward run (checkpoints every `every`
              steps), reverse sweep of a final-state gradient, gradient out
"""
import functools
import math

import numpy as np
import torch

import nebulasem_gb300 as ng
from nebulasem_gb300 import mesh as ngmesh
from nebulasem_gb300 import objective

P0, T0, CP, CV, GRAV, PR = 1e5, 300.0, 1004.5, 717.5, 9.81, 0.9


def _case(kind, n, order, h, steps=1, dim=3, tilt=0.0, visc=0.0, prec="mixed", every=0):
    return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], order=order, h=h, dim=dim, tilt=tilt,
                visc=visc, prec=prec, steps=steps, every=every)


def listed():
    out = {
        # one right-hand side of the small 2D bubble: a host time integrator's
        # own call, all latency
        "tendency_2d_10x10_n4": _case("tendency", (10, 1, 10), 4, 100.0, dim=2),
        # the 2D rising bubble of the reference's srtb example, stepped
        "mixed_2d_10x10_n4": _case("step", (10, 1, 10), 4, 100.0, steps=50, dim=2),
        # a small 3D box with ragged element counts: less than one wave of CTAs
        "mixed_3d_9x7x11_n4": _case("step", (9, 7, 11), 4, 62.5, steps=40),
        # the 32^3 bubble: the benchmark's workload
        "mixed_3d_32_n4": _case("step", (32, 32, 32), 4, 62.5, steps=40),
        # order 7: fewer, larger elements
        "mixed_3d_16_n7": _case("step", (16, 16, 16), 7, 125.0, steps=30),
        # artificial viscosity (diffusion YES), ragged box
        "mixed_visc_20x21x22_n4": _case("step", (20, 21, 22), 4, 62.5, steps=20, visc=1.5),
        # inclined elements: the full-metric kernels
        "mixed_tilt_24x15x19_n4": _case("step", (24, 15, 19), 4, 62.5, steps=20, tilt=30.0),
        # the parity form
        "fp64_3d_14x12x13_n4": _case("step", (14, 12, 13), 4, 62.5, steps=10, prec="fp64"),
        # the reference's segregated update, 2D with viscosity, as its examples
        "segregated_2d_32x24_n4_visc": _case("segregated", (32, 1, 24), 4, 50.0, steps=40, dim=2,
                                             visc=1.5, prec="fp64"),
        # scalar convection by a fixed wind, order 5
        "convection_12x14x10_n5": _case("convection", (12, 14, 10), 5, 62.5, steps=40,
                                        prec="fp64"),
        # gradient of a final-state objective in each form
        "adjoint_mixed_16_n4": _case("adjoint", (16, 16, 16), 4, 125.0, steps=20, every=10),
        "adjoint_fp64_9x8x10_n4": _case("adjoint", (9, 8, 10), 4, 125.0, steps=8, every=4,
                                        prec="fp64"),
    }
    return [dict(c, name=k) for k, c in out.items()]


def draw(rng):
    """One more case of the ranges above: element counts spread over their
    logarithm and unequal per direction, orders the form is built for."""
    def box(lo, hi, dim=3):
        """Unequal counts with a product between lo and hi (log-uniform)."""
        total = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        side = total ** (1.0 / dim)
        a = max(2, round(side * rng.uniform(0.75, 1.3)))
        b = max(2, round(side * rng.uniform(0.75, 1.3))) if dim == 3 else 1
        c = max(2, math.ceil(total / (a * b)))
        while a * b * c > hi and c > 2:
            c -= 1
        return a, b, c

    h = rng.choice([50.0, 62.5, 100.0, 125.0])
    visc = rng.choice([0.0, 1.5])
    kind = rng.choice(["tendency", "mixed", "mixed", "mixed2d", "mixed_n7", "mixed_tilt", "fp64",
                       "segregated", "convection", "adjoint_mixed", "adjoint_fp64"])
    if kind == "tendency":
        if rng.random() < 0.5:
            return _case("tendency", box(64, 1024, 2), rng.choice([3, 4]), h, dim=2)
        return _case("tendency", box(64, 2048), rng.choice([3, 4, 7]), h)
    if kind == "mixed2d":
        return _case("step", box(64, 8192, 2), rng.choice([3, 4]), h, steps=rng.randint(20, 60),
                     dim=2, visc=visc)
    if kind == "mixed":
        return _case("step", box(64, 20000), rng.choice([3, 4]), h, steps=rng.randint(10, 40),
                     visc=visc)
    if kind == "mixed_n7":
        return _case("step", box(64, 3000), 7, h, steps=rng.randint(10, 25), visc=visc)
    if kind == "mixed_tilt":
        return _case("step", box(64, 6000), rng.choice([3, 4]), h, steps=rng.randint(10, 20),
                     tilt=rng.choice([15.0, 30.0, 45.0]), visc=visc)
    if kind == "fp64":
        return _case("step", box(27, 1500), rng.choice([3, 4, 5]), h, steps=rng.randint(3, 8),
                     visc=visc, prec="fp64")
    if kind == "segregated":
        if rng.random() < 0.6:
            return _case("segregated", box(64, 2048, 2), rng.choice([3, 4]), h,
                         steps=rng.randint(10, 40), dim=2, visc=visc, prec="fp64")
        return _case("segregated", box(27, 600), rng.choice([3, 4]), h, steps=rng.randint(5, 15),
                     visc=visc, prec="fp64")
    if kind == "convection":
        return _case("convection", box(64, 2000), rng.choice([3, 4, 5]), h,
                     steps=rng.randint(10, 40), prec="fp64")
    if kind == "adjoint_mixed":
        return _case("adjoint", box(64, 4096), rng.choice([3, 4]), h, steps=rng.randint(8, 16),
                     every=rng.choice([4, 5, 8]))
    return _case("adjoint", box(27, 700), rng.choice([3, 4]), h, steps=rng.randint(3, 8),
                 every=rng.choice([2, 3, 4]), prec="fp64")


def _dt(case):
    """Stable step: 0.0075 s at h = 62.5 m, N = 4, scaled with h / N^2."""
    dt = 0.0075 * (case["h"] / 62.5) * 16.0 / case["order"] ** 2
    return 0.5 * dt if case["kind"] == "segregated" else dt   # forward Euler


@functools.lru_cache(maxsize=2)
def _mesh(nx, ny, nz, order, h, dim, tilt):
    """Mesh and hydrostatic background in the reference's layout (no seed in it)."""
    m = ngmesh.box_mesh((nx, ny, nz), order, (nx * h, ny * h, nz * h), dim=dim, tilt=tilt)
    _, m["p_ref"], m["rho_ref"], m["gh"] = ngmesh.bubble_state(m, 0.0, (0.0,) * 3, (1.0,) * 3)
    return m


def _case_mesh(case):
    return _mesh(case["nx"], case["ny"], case["nz"], case["order"], case["h"], case["dim"],
                 case["tilt"])


def _inputs(case, seed):
    """Mesh and initial conserved state: a bubble of drawn amplitude, centre and
    radius (p' = 0), moved by three smooth wind modes."""
    m = _case_mesh(case)
    rng = np.random.default_rng(seed)
    n_int = int(m["meta"][7])
    x = np.asarray(m["cC"]).reshape(-1, 3)[:n_int]
    lo, hi = x.min(axis=0), x.max(axis=0)
    size = np.maximum(hi - lo, 1.0)
    amp = rng.uniform(0.3, 0.7)
    centre = lo + size * rng.uniform(0.4, 0.6, 3)
    r = (x - centre) / (size.min() if case["dim"] == 3 else min(size[0], size[2]))
    if case["dim"] == 2:
        r[:, 1] = 0.0
    r = np.minimum(1.0, np.sqrt((r ** 2).sum(axis=1)) / rng.uniform(0.25, 0.4))
    theta_p = 0.5 * amp * (1.0 + np.cos(np.pi * r))
    u = objective.state_from_theta(theta_p, m["p_ref"][:n_int], P0, T0, CP, CV)
    y = (x - lo) / size
    for _ in range(3):
        k = rng.integers(1, 4, 3) * np.pi
        mode = np.sin(y @ k + rng.uniform(0, 2 * np.pi))
        for c in (0, 1, 2) if case["dim"] == 3 else (0, 2):
            u[1 + c] += u[0] * mode * rng.uniform(-0.35, 0.35)
    return m, u, theta_p


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t.numpy()


def _lam(case, m, u):
    """Gradient of 1/2 sum theta'^2 over a box of the upper half of the domain
    with respect to the state."""
    n_int = int(m["meta"][7])
    x = np.asarray(m["cC"]).reshape(-1, 3)[:n_int]
    lo, hi = x.min(axis=0), x.max(axis=0)
    w = hi - lo
    mask = objective.box_mask(x, (lo[0] + 0.3 * w[0], lo[0] + 0.7 * w[0],
                                  lo[2] + 0.5 * w[2], lo[2] + 0.9 * w[2]))
    return objective.objective_grad(u, mask, T0)


def _wind(u):
    """The convection cases' wind: a uniform one plus the state's modes."""
    w = np.stack([u[1] / u[0] + 6.0, u[2] / u[0] - 4.0, u[3] / u[0] + 5.0], axis=1)
    return np.ascontiguousarray(w)


def prepare(case, seed):
    m, u, theta_p = _inputs(case, seed)
    s = ng.Solver(m, dt=_dt(case), viscosity=case["visc"], Pr=PR)
    st = {"case": case, "solver": s}
    if case["kind"] == "segregated":
        st["rho"], st["T"] = _pinned(u[0]), _pinned(theta_p)
        st["U"] = _pinned(np.stack([u[1] / u[0], u[2] / u[0], u[3] / u[0]], axis=1))
        return st
    if case["kind"] == "convection":
        st["U"], st["T"] = _wind(u), theta_p.copy()
        return st
    st["in"] = (_pinned(u[0]), _pinned(np.stack(u[1:4], axis=1)), _pinned(u[4]))
    st["out"] = tuple(_pinned(np.zeros_like(a)) for a in st["in"])
    if case["kind"] == "adjoint":
        st["lam"] = _lam(case, m, u)
    return st


def run(state):
    case, s = state["case"], state["solver"]
    prec = ng.FP64 if case["prec"] == "fp64" else ng.MIXED
    kind = case["kind"]
    if kind == "segregated":
        s.set_fields(state["rho"], state["U"], state["T"])
        s.step(case["steps"], prec=ng.FP64, sync=False, scheme=ng.REF_SEGREGATED)
        return s.get_fields()
    if kind == "convection":
        s.convection_set(state["U"], state["T"])
        s.convection_step(case["steps"])
        return s.convection_get()
    s.set_state_raw(*state["in"])
    if kind == "tendency":
        return s.tendency(prec)
    if kind == "step":
        s.step(case["steps"], prec=prec, sync=False)
        s.get_state_raw(*state["out"])
        return state["out"]
    s.forward_checkpointed(case["steps"], case["every"], prec)
    lam0, _ = s.adjoint(state["lam"])
    return lam0


def work(case):
    """Bytes: the state (the wind and the scalar for convection; the state and
    the adjoint state for the adjoint) read once and the result written once.
    Flops: per node and right-hand side the line sums, the pointwise physics and
    the faces' share of the Rusanov fluxes; the adjoint counts the forward, its
    recomputation and a transposed pass."""
    n = case["order"] + 1
    dirs = 3 if case["dim"] == 3 else 2
    nodes = case["nx"] * case["ny"] * case["nz"] * n ** dirs
    nv = 1 if case["kind"] == "convection" else 5
    rhs = 3 if case["kind"] in ("step", "adjoint") else 1
    faces = 2 * dirs / n
    flops = nv * dirs * 2 * n + (14 * nv + 25 if nv == 5 else 6) + faces * 12 * nv
    if case["visc"]:
        flops += 4 * dirs * 2 * n + 60
    if case["tilt"]:
        flops += nv * dirs * 5
    passes = 3.0 if case["kind"] == "adjoint" else 1.0
    values = {"convection": 4 + 1, "adjoint": 10 + 5}.get(case["kind"], 5 + 5)
    return {"bytes": nodes * 8.0 * values, "flops": nodes * flops * rhs * case["steps"] * passes}


# ----------------------------------------------------------------- 64 bits

class _Box:
    """The same equations in plain torch float64 on a box of equal elements:
    weak-form spectral-element divergence with Rusanov fluxes, arrays
    [nx, ny, nz, NPX, NPY, NPZ] per variable."""

    def __init__(self, case, m):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        meta = [int(v) for v in m["meta"]]
        self.shape = (case["nx"], case["ny"], case["nz"], meta[0], meta[1], meta[2])
        self.dirs = [d for d in range(3) if self.shape[3 + d] > 1]
        h = case["h"]
        self.J = 2.0 / h
        ang = math.radians(case["tilt"])
        c, s = math.cos(ang), math.sin(ang)
        self.R = [[c, 0.0, s], [0.0, 1.0, 0.0], [-s, 0.0, c]]   # R[r][d]
        self.Q, self.D, self.wend = {}, {}, {}
        for d in self.dirs:
            n = self.shape[3 + d]
            dp = torch.tensor(np.asarray(m[f"dpsi{d}"]).reshape(n, n), dtype=torch.float64,
                              device=self.dev)                  # [s][i] = l_i'(x_s)
            w = torch.tensor(np.asarray(m[f"wgl{d}"]), dtype=torch.float64, device=self.dev)
            self.Q[d] = dp.T * w[None, :] / w[:, None]
            self.D[d] = dp
            self.wend[d] = float(w[0])
        self.nu = case["visc"]
        self.g = (0.0, 0.0, -GRAV)
        n_int = meta[7]
        self.p_ref = self.field(m["p_ref"][:n_int])
        self.rho_ref = self.field(m["rho_ref"][:n_int])
        self.Rgas, self.gam = CP - CV, CP / CV

    def field(self, a):
        a = np.ascontiguousarray(np.asarray(a, dtype=np.float64))
        return torch.tensor(a, device=self.dev).reshape(self.shape)

    @staticmethod
    def flat(t):
        return t.reshape(-1).cpu().numpy()

    def along(self, M, q, d):
        return (q.movedim(3 + d, -1) @ M.T).movedim(-1, 3 + d)

    @staticmethod
    def norm(v):
        s = v[0] * v[0] + v[1] * v[1] + v[2] * v[2]
        pos = s > 0
        return torch.where(pos, torch.where(pos, s, torch.ones_like(s)).sqrt(),
                           torch.zeros_like(s))

    def pressure(self, rt):
        return P0 * (rt * (self.Rgas / P0)) ** self.gam - self.p_ref

    def lower(self, q, d):
        return q.select(3 + d, 0)

    def upper(self, q, d):
        return q.select(3 + d, self.shape[3 + d] - 1)

    def ghost(self, U, en):
        un = sum(U[r] * en[r] for r in range(3))
        t = [U[r] - un * en[r] for r in range(3)]
        mt = self.norm(t)
        big = mt > 1e-7
        sc = torch.where(big, self.norm(U) / torch.where(big, mt, torch.ones_like(mt)),
                         torch.ones_like(mt))
        return [x * sc for x in t]

    def add_faces(self, L, d, face_flux, coef):
        """L -= coef F_out at the end nodes of every line of direction d;
        face_flux(minus, plus) is the flux along +d between the elements and
        face_flux(.., None) / (None, ..) that of the upper / lower wall, each
        given the slice of elements on its side."""
        n_el = self.shape[d]
        hi = [face_flux(slice(0, n_el - 1), slice(1, n_el))] if n_el > 1 else []
        up = face_flux(slice(n_el - 1, n_el), None)
        low = face_flux(None, slice(0, 1))
        out = []
        for v in range(len(L)):
            inner = [hi[0][v]] if hi else []
            F_up = torch.cat(inner + [up[v]], dim=d)
            F_lo = torch.cat([low[v]] + inner, dim=d)
            n = self.shape[3 + d]
            z = torch.zeros_like(L[v]).movedim(3 + d, -1)
            parts = [coef * F_lo.unsqueeze(-1), z[..., 1:n - 1], -coef * F_up.unsqueeze(-1)]
            out.append(L[v] + torch.cat(parts, dim=-1).movedim(-1, 3 + d))
        return out

    def gradients(self, U, th):
        """G[r][c] = d_r U_c (c < 3), d_r theta (c = 3): strong form with the
        face terms (average - own) along the outward normal."""
        q = list(U) + [th]
        G = [[torch.zeros_like(th) for _ in range(4)] for _ in range(3)]
        for d in self.dirs:
            dq = [self.J * self.along(self.D[d], x, d) for x in q]
            en = [self.R[r][d] for r in range(3)]
            n_el = self.shape[d]
            lift = []
            lo = [self.lower(x, d) for x in q]
            up = [self.upper(x, d) for x in q]
            gl = self.ghost([x.narrow(d, 0, 1) for x in lo[:3]], en) + [lo[3].narrow(d, 0, 1)]
            gu = self.ghost([x.narrow(d, n_el - 1, 1) for x in up[:3]], en) + \
                [up[3].narrow(d, n_el - 1, 1)]
            for c in range(4):
                mid = 0.5 * (up[c].narrow(d, 0, n_el - 1) + lo[c].narrow(d, 1, n_el - 1))
                at_lo = torch.cat([gl[c], mid], dim=d) - lo[c]
                at_up = torch.cat([mid, gu[c]], dim=d) - up[c]
                lift.append((at_lo, at_up))
            k = self.J / self.wend[d]
            for c in range(4):
                x = dq[c].movedim(3 + d, -1).clone()
                x[..., 0] -= k * lift[c][0]
                x[..., -1] += k * lift[c][1]
                x = x.movedim(-1, 3 + d)
                for r in range(3):
                    if en[r]:
                        G[r][c] = G[r][c] + en[r] * x
        return G

    def divergence(self, flux, state, lam_of, walls, mom_row=None):
        """-(weak divergence) of the vectors flux[v] (three components each)
        with Rusanov faces: the jumps of state[v], and of the three momentum
        rows from mom_row on only their component along the normal."""
        L = [torch.zeros_like(self.p_ref) for _ in flux]
        for d in self.dirs:
            en = [self.R[r][d] for r in range(3)]
            Fn = [sum(en[c] * f[c] for c in range(3) if en[c]) for f in flux]
            L = [x + self.J * self.along(self.Q[d], f, d) for x, f in zip(L, Fn)]
            lo = [self.lower(f, d) for f in Fn]
            up = [self.upper(f, d) for f in Fn]
            sl = [self.lower(x, d) for x in state]
            su = [self.upper(x, d) for x in state]
            spd_l, spd_u = self.lower(lam_of, d), self.upper(lam_of, d)

            def face(minus, plus):
                if minus is None or plus is None:
                    side, sg = (plus, -1.0) if minus is None else (minus, 1.0)
                    pick = (lambda q: self.cut(self.lower(q, d), d, side)) if minus is None \
                        else (lambda q: self.cut(self.upper(q, d), d, side))
                    return walls(pick, en, sg)
                lam = 0.25 * (self.cut(spd_u, d, minus) + self.cut(spd_l, d, plus))
                j = [self.cut(b, d, plus) - self.cut(a, d, minus) for a, b in zip(su, sl)]
                av = [0.5 * (self.cut(a, d, minus) + self.cut(b, d, plus)) for a, b in zip(up, lo)]
                if mom_row is not None:
                    o = mom_row
                    jn = sum(en[r] * j[o + r] for r in range(3) if en[r])
                    for r in range(3):
                        j[o + r] = en[r] * jn
                return [a - lam * x for a, x in zip(av, j)]

            L = self.add_faces(L, d, face, self.J / self.wend[d])
        return L

    @staticmethod
    def cut(q, d, sl):
        return q.narrow(d, sl.start, sl.stop - sl.start)

    def wall_momentum(self, pick, en, sg, pp, mom, U, cs):
        """Momentum flux along +en of a wall whose outward normal is sg en:
        p' n plus the Rusanov term of the normal momentum."""
        Uw = [pick(x) for x in U]
        lam = 0.5 * (self.norm(self.ghost(Uw, en)) + pick(cs))
        mn = sum(en[r] * pick(mom[r]) for r in range(3) if en[r])
        f = pick(pp) + sg * lam * mn
        return [en[r] * f for r in range(3)]

    def rhs(self, u):
        rho, mom, rt = u[0], u[1:4], u[4]
        U = [x / rho for x in mom]
        th = rt / rho
        pp = self.pressure(rt)
        cs = (self.gam * self.Rgas * th).sqrt()
        flux = [mom, *self.momentum_flux(mom, U, pp), [x * th for x in mom]]
        if self.nu:
            self.add_viscous(flux[1:4], flux[4], rho * self.nu, self.gradients(U, th))

        def walls(pick, en, sg):
            z = torch.zeros_like(pick(rho))
            return [z, *self.wall_momentum(pick, en, sg, pp, mom, U, cs), z]

        L = self.divergence(flux, u, self.norm(U) + cs, walls, mom_row=1)
        for r in range(3):
            if self.g[r]:
                L[1 + r] = L[1 + r] + (rho - self.rho_ref) * self.g[r]
        return L

    @staticmethod
    def momentum_flux(mom, U, pp):
        return [[mom[r] * U[c] + (pp if r == c else 0.0) for c in range(3)] for r in range(3)]

    @staticmethod
    def add_viscous(mflux, tflux, mu, G):
        for r in range(3):
            for c in range(3):
                mflux[r][c] = mflux[r][c] - mu * G[r][c]
        for c in range(3):
            tflux[c] = tflux[c] - (mu / PR) * G[c][3]

    def step(self, u, dt):
        u1 = [a + dt * b for a, b in zip(u, self.rhs(u))]
        u2 = [0.75 * a + 0.25 * (b + dt * c) for a, b, c in zip(u, u1, self.rhs(u1))]
        return [a / 3 + 2.0 / 3.0 * (b + dt * c) for a, b, c in zip(u, u2, self.rhs(u2))]

    def segregated_step(self, rho, U, tp, dt):
        th = tp + T0
        mom = [rho * x for x in U]
        cs = (self.gam * self.Rgas * th).sqrt()
        spd = self.norm(U) + cs
        zero = lambda pick, en, sg: [torch.zeros_like(pick(rho))]
        rho1 = rho + dt * self.divergence([mom], [rho], spd, zero)[0]
        pp = self.pressure(rho1 * th)
        mflux, tflux = self.momentum_flux(mom, U, pp), [x * th for x in mom]
        if self.nu:
            self.add_viscous(mflux, tflux, rho * self.nu, self.gradients(U, th))
        mom1 = [rho1 * x for x in U]
        Lm = self.divergence(mflux, mom1, spd,
                             lambda pick, en, sg: self.wall_momentum(pick, en, sg, pp, mom1, U, cs),
                             mom_row=0)
        for r in range(3):
            if self.g[r]:
                Lm[r] = Lm[r] + (rho1 - self.rho_ref) * self.g[r]
        Lt = self.divergence([tflux], [rho1 * th], spd, zero)[0]
        U1 = [(a + dt * b) / rho1 for a, b in zip(mom, Lm)]
        return rho1, U1, (rho * th + dt * Lt) / rho1 - T0

    def convection_step(self, U, T, dt):
        zero = lambda pick, en, sg: [torch.zeros_like(pick(T))]
        return T + dt * self.divergence([[x * T for x in U]], [T], self.norm(U), zero)[0]


def exact(case, seed):
    m, u, theta_p = _inputs(case, seed)
    b = _Box(case, m)
    dt = _dt(case)
    with torch.no_grad():
        x = [b.field(a) for a in u]
        if case["kind"] == "tendency":
            return [b.flat(a) for a in b.rhs(x)]
        if case["kind"] == "convection":
            w = _wind(u)
            U, T = [b.field(w[:, c]) for c in range(3)], b.field(theta_p)
            for _ in range(case["steps"]):
                T = b.convection_step(U, T, dt)
            return b.flat(T)
        if case["kind"] == "segregated":
            f = (x[0], [b.field(u[1 + c] / u[0]) for c in range(3)], b.field(theta_p))
            for _ in range(case["steps"]):
                f = b.segregated_step(*f, dt)
            return (b.flat(f[0]), np.stack([b.flat(a) for a in f[1]], axis=1), b.flat(f[2]))
        traj = [x]
        for _ in range(case["steps"]):
            x = b.step(x, dt)
            if case["kind"] == "adjoint":
                traj.append(x)
        if case["kind"] == "step":
            return (b.flat(x[0]), np.stack([b.flat(a) for a in x[1:4]], axis=1), b.flat(x[4]))
    lam = [b.field(a) for a in _lam(case, m, u)]
    for x in reversed(traj[:-1]):
        x = [a.detach().requires_grad_(True) for a in x]
        y = b.step(x, dt)
        lam = [a.detach() for a in torch.autograd.grad(y, x, lam)]
    return [b.flat(a) for a in lam]
