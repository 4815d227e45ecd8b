"""The work a user of libsph_b200 has it do, as cases that can be timed and checked.

A case is a dict of plain values.  `prepare` builds what a host program holds
before the call (the handle with its uploaded state, page-locked output arrays),
`run` is one pass through the public entry points of sph-2d_b200/sph_b200.py, and
`exact` restates the same pass in FP64 torch, without the library.

Kinds
  run      time_iteration(steps) on the device-resident state, then the new x, v
           and rho delivered to page-locked host arrays (the output interval of a
           production run).  Later passes go on from where the last one stopped.
  coupled  one step of a host that owns its arrays: update_state, one step, get_state
  rhs      single_step_compute: one right-hand side, its rates and flags returned
  pairs    find_particle_pair with kernel values and gradients, through the C entry
           into the arrays a Fortran host sizes once
  adjoint  one evaluation of an optimisation loop: set_state, the checkpointed
           forward run, the gradient with respect to the initial state and nu
The flow is "tgv" (Taylor-Green vortex, periodic box) or "square" (moving square in
a tank, ghost assignment and body force at every right-hand side).  Initial states
carry a seeded jitter of +-0.1 dx (tank water: +-0.05 dx).
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sph-2d_b200"))
import sph_b200 as S  # noqa: E402

SOLVERS = {"modlr": S.SOLVER_MODLR_DELTA_SPS, "muscl": S.SOLVER_MUSCL_DELTA_SPS, "plain": S.SOLVER_DELTA_SPS,
           "ms_modlr": S.SOLVER_MS_MODLR_DELTA, "ms_hllc": S.SOLVER_MS_HLLC_DELTA}
PRECISION = {"fp64": S.PREC_FP64, "mixed": S.PREC_MIXED}


def listed():
    return [
        # the smallest call: a host that edits its arrays each step (47 x 47 particles)
        {"name": "coupled_47_fp64", "kind": "coupled", "flow": "tgv", "side": 47, "solver": "muscl",
         "precision": "fp64", "shipped": False},
        # the 100 x 100 Taylor-Green case with the plain method, ten steps an output
        {"name": "run_100_plain_fp64", "kind": "run", "flow": "tgv", "side": 100, "solver": "plain",
         "precision": "fp64", "shipped": False, "steps": 10},
        # the Taylor-Green case as the reference ships it (Gaussian kernel, quadratic MLS every 20 steps)
        {"name": "run_100_shipped_fp64", "kind": "run", "flow": "tgv", "side": 100, "solver": "modlr",
         "precision": "fp64", "shipped": True, "steps": 20},
        # an ordinary run of a size nobody tuned for
        {"name": "run_401_muscl_mixed", "kind": "run", "flow": "tgv", "side": 401, "solver": "muscl",
         "precision": "mixed", "shipped": False, "steps": 5},
        # the benchmark's 2048 x 2048 case, in both precisions
        {"name": "run_2048_muscl_mixed", "kind": "run", "flow": "tgv", "side": 2048, "solver": "muscl",
         "precision": "mixed", "shipped": False, "steps": 5},
        {"name": "run_2048_muscl_fp64", "kind": "run", "flow": "tgv", "side": 2048, "solver": "muscl",
         "precision": "fp64", "shipped": False, "steps": 3},
        # the moving square at D/100 (512,064 particles), HLLC, mixed; and a coarse FP64 tank with the
        # solver the moving-square case ships
        {"name": "square_100_hllc_mixed", "kind": "run", "flow": "square", "per_d": 100, "solver": "ms_hllc",
         "precision": "mixed", "steps": 10},
        {"name": "square_30_modlr_fp64", "kind": "run", "flow": "square", "per_d": 30, "solver": "ms_modlr",
         "precision": "fp64", "steps": 10},
        # the drop-in of single_step_compute and of find_particle_pair for a Fortran host
        {"name": "rhs_257_muscl_fp64", "kind": "rhs", "flow": "tgv", "side": 257, "solver": "muscl",
         "precision": "fp64", "shipped": False},
        {"name": "pairs_300_fp64", "kind": "pairs", "flow": "tgv", "side": 300, "solver": "modlr",
         "precision": "fp64", "shipped": False},
        # gradients: the 256 x 256 velocity misfit with a checkpoint every 32 steps (two segments of it),
        # and the drag impulse of a coarse tank
        {"name": "adjoint_256_mixed", "kind": "adjoint", "flow": "tgv", "side": 256, "solver": "modlr",
         "precision": "mixed", "shipped": False, "steps": 64, "every": 32},
        {"name": "adjoint_square_25_fp64", "kind": "adjoint", "flow": "square", "per_d": 25, "solver": "ms_modlr",
         "precision": "fp64", "steps": 32, "every": 16},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["run", "run", "run", "square", "square", "coupled", "rhs", "pairs", "adjoint", "adjoint_square"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "run":
        if rng.random() < 0.25:
            return {"kind": "run", "flow": "tgv", "side": size(50, 400), "solver": "modlr", "precision": prec,
                    "shipped": True, "steps": rng.randint(1, 20)}
        side = size(40, 2000)
        return {"kind": "run", "flow": "tgv", "side": side, "solver": rng.choice(["muscl", "muscl", "modlr", "plain"]),
                "precision": prec, "shipped": False, "steps": rng.randint(1, 3 if side > 800 else 12)}
    if kind == "square":
        return {"kind": "run", "flow": "square", "per_d": size(12, 100), "solver": rng.choice(["ms_hllc", "ms_modlr"]),
                "precision": prec, "steps": rng.randint(1, 12)}
    if kind == "coupled":
        return {"kind": "coupled", "flow": "tgv", "side": size(24, 600), "solver": rng.choice(["muscl", "modlr"]),
                "precision": prec, "shipped": False}
    if kind == "rhs":
        return {"kind": "rhs", "flow": "tgv", "side": size(40, 600), "solver": rng.choice(["muscl", "modlr", "plain"]),
                "precision": "fp64", "shipped": rng.random() < 0.3}
    if kind == "pairs":
        return {"kind": "pairs", "flow": "tgv", "side": size(30, 500), "solver": "modlr", "precision": prec,
                "shipped": rng.random() < 0.5}
    every = rng.choice([4, 8, 16])
    steps = every * rng.randint(1, 2) - rng.randint(0, 1)
    if kind == "adjoint":
        return {"kind": "adjoint", "flow": "tgv", "side": size(32, 256), "solver": rng.choice(["modlr", "muscl", "plain"]),
                "precision": prec, "shipped": False, "steps": steps, "every": every}
    return {"kind": "adjoint", "flow": "square", "per_d": size(10, 30), "solver": rng.choice(["ms_modlr", "ms_hllc"]),
            "precision": prec, "steps": steps, "every": every}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dt(cfg):
    return 0.25 * cfg.h / math.sqrt(cfg.c0sq) if cfg.integrator == S.INTEGRATOR_EULER_PC else S.baseline_dt(cfg)


def _inputs(case, seed):
    """(TgvCase, initial types, wall labels, adjoint target or None) of a case."""
    prec = PRECISION[case["precision"]]
    if case["flow"] == "square":
        c, ity = S.make_moving_square(dx=1.0 / case["per_d"], lx=10.0, ly=5.0, D=1.0, U=1.0,
                                      solver=SOLVERS[case["solver"]], precision=prec, jitter=0.05, seed=seed)
        c.cfg.ghost_assign = 1
        if case["kind"] == "adjoint":
            c.cfg.mls_order = 0
        return c, ity, S.moving_square_labels(c, ity), None
    c = S.make_tgv(case["side"], reference=case["shipped"], solver=SOLVERS[case["solver"]], precision=prec,
                   jitter=0.1, seed=seed)
    c.cfg.precision = prec
    target = None
    if case["kind"] == "adjoint":
        target = c.vel + S.fourier_perturbation(c.pos, n_modes=8, amp=0.05, seed=seed + 1)
    return c, None, None, target


def _pair_cap(c):
    """Length of a host's pair arrays: the lattice count in the support plus a margin."""
    r = c.cfg.kernel_scale * c.cfg.h / c.cfg.dx
    return int(c.n * (0.5 * math.pi * r * r * 1.2 + 4)) + 4096


def _upload(st):
    c = st["c"]
    st["sim"].set_state(c.pos, c.vel, c.rho, c.mass, c.type)
    if st["ity"] is not None:
        st["sim"].set_initial_type(st["ity"])
        st["sim"].set_boundary_labels(st["lab"])
        st["sim"].set_body_motion((1.0, 0.0))


def prepare(case, seed):
    c, ity, lab, target = _inputs(case, seed)
    st = {"case": case, "c": c, "ity": ity, "lab": lab, "target": target, "dt": _dt(c.cfg),
          "sim": S.Simulation(c.cfg, c.n)}
    _upload(st)
    if case["kind"] == "run":
        st["out"] = [torch.empty(m * c.n, dtype=torch.float64).pin_memory().numpy() for m in (2, 2, 1)]
    if case["kind"] == "pairs":
        cap = _pair_cap(c)
        st["pairs"] = [np.zeros(cap, np.int32), np.zeros(cap, np.int32), np.zeros(cap), np.zeros(2 * cap)]
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    sim, case, c = st["sim"], st["case"], st["c"]
    kind = case["kind"]
    if kind == "run":
        d = sim.time_iteration(case["steps"], st["dt"])
        pos, vel, rho = st["out"]
        sim.snapshot_begin(pos, vel, rho, None)
        sim.snapshot_wait()
        out = {"pos": pos, "vel": vel, "rho": rho, "kinetic_energy": d.kinetic_energy}
        if case["flow"] == "square":
            out["body_force"] = np.array(d.body_force[:])
        return out
    if kind == "coupled":
        sim.update_state(c.pos, c.vel, c.rho)
        sim.time_iteration(1, st["dt"])
        pos, vel, rho, _ = sim.get_state()
        return {"pos": pos, "vel": vel, "rho": rho}
    if kind == "rhs":
        return sim.single_step_compute()
    if kind == "pairs":
        pi, pj, w, dw = st["pairs"]
        count = ctypes.c_longlong(0)
        ip, dp = ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_double)
        code = sim.lib.sph_find_particle_pair(sim.h, pi.size, pi.ctypes.data_as(ip), pj.ctypes.data_as(ip),
                                              w.ctypes.data_as(dp), dw.ctypes.data_as(dp), ctypes.byref(count))
        if code != S.SPH_OK:
            raise S.SphError(code, "sph_find_particle_pair")
        return {"pair_i": pi, "pair_j": pj, "w": w, "dwdx": dw, "pair_number": count.value}
    _upload(st)
    drag = case["flow"] == "square"
    loss = sim.adjoint_forward(case["steps"], st["dt"], checkpoint_every=case["every"],
                               loss=S.LOSS_DRAG if drag else S.LOSS_VELOCITY_MISFIT, target_vel=st["target"])
    out = dict(sim.adjoint_backward(1.0), loss=loss)
    if drag:
        out["motion"] = sim.adjoint_motion_gradient()
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the state (x, v, rho, mass, type) read once and what is returned
    written once.  Operations: per right-hand side and interacting pair (each
    pair once) the terms of the solver, about 60 operations for pass-A sums
    (kernel, tensor, gradients) and 150 for the forces, 60 more for the MUSCL
    or HLLC state; an adjoint step about three forward ones."""
    if case["flow"] == "square":
        n = int(50 * case["per_d"] ** 2 + 8 * 15 * case["per_d"])
        pairs = 0.5 * math.pi * 3.45 ** 2 * n
        rhs_per_step, ops = 1, 210 + (60 if case["solver"] == "ms_hllc" else 0)
    else:
        n = case["side"] ** 2
        r = 3.6 if case["shipped"] else 2.6
        pairs = 0.5 * math.pi * r * r * n
        rhs_per_step, ops = 3, 210 + (60 if case["solver"] == "muscl" else 0)
    state = n * (5 * 8 + 8 + 4)
    kind = case["kind"]
    if kind == "pairs":
        return {"bytes": n * 20 + pairs * 32, "flops": pairs * 20}
    if kind == "rhs":
        return {"bytes": state + n * (5 * 8 + 2 * 4), "flops": pairs * ops}
    flops = case.get("steps", 1) * rhs_per_step * pairs * ops
    if kind == "adjoint":
        return {"bytes": state + n * 5 * 8, "flops": 4 * flops}
    return {"bytes": state + n * 5 * 8, "flops": flops}


# ---------------------------------------------------------------------------
# the same in FP64 torch, from the equations
# ---------------------------------------------------------------------------
class _Consts:
    """Constants of a configuration; the shipped cases use default-real literals."""

    def __init__(self, c):
        f = np.float32
        q = bool(c.reference_literals)
        self.c, self.q = c, q
        self.gauss = c.kernel_model == S.KERNEL_GAUSSIAN
        pi_k = float(f(3.14159265358)) if q else math.pi
        e9 = f(np.exp(f(-9.0)))
        self.e9 = float(e9) if q else math.exp(-9.0)
        den = float(f(1.0) - f(10.0) * e9) if q else 1.0 - 10.0 * self.e9
        self.kf = lambda h: 1.0 / (pi_k * h * h * den) if self.gauss else 7.0 / (4 * pi_k * h * h)
        self.cut_min = float(f(1.0e-7)) if q else 1.0e-7
        self.sps_dl = (float(np.sqrt(f(2.0)) / f(2.0)) if q else math.sqrt(2.0) / 2.0) * c.dx
        self.c012 = float(f(0.12)) if q else 0.12
        self.c23 = float(f(2.0) / f(3.0)) if q else 2.0 / 3.0
        self.blin = float(f(2.0) / f(3.0) * f(0.0066)) if q else 2.0 / 3.0 * 0.0066
        self.r = c.kernel_scale * c.h
        self.ghost_h = (float(f(c.ghost_h_factor)) if q else c.ghost_h_factor) * c.h

    def kernel(self, d, h):
        """W and (dW/dd)/d at distance d."""
        q, kf = d / h, self.kf(h)
        if self.gauss:
            e = torch.exp(-q * q)
            return (e - self.e9) * kf, -2.0 * e * kf / (h * h)
        t = 1.0 - 0.5 * q
        return kf * (1.0 + 2.0 * q) * t ** 4, -5.0 * kf * t ** 3 / (h * h)

    def eos(self, rho):
        c = self.c
        r = rho / c.rho0
        p = c.c0sq * c.rho0 / 7.0 * (r ** 7 - 1.0) if c.eos == S.EOS_TAIT else c.c0sq * (rho - c.rho0)
        return p + c.background_p, math.sqrt(c.c0sq) * r ** 3


def _near(x, y, radius, keep, targets=None):
    """Ordered pairs (a, b), a != b, with |x_a - x_b| <= radius; keep(a, b) says which types meet."""
    with torch.no_grad():
        x, y = x.detach(), y.detach()
        n = x.numel()
        cx, cy = ((x - x.min()) / radius).long() + 1, ((y - y.min()) / radius).long() + 1
        nx, ny = int(cx.max()) + 2, int(cy.max()) + 2
        key = cy * nx + cx
        order = torch.argsort(key, stable=True)
        count = torch.bincount(key, minlength=nx * ny)
        start = torch.cumsum(count, 0) - count
        who = torch.arange(n, device=x.device) if targets is None else targets
        pa, pb = [], []
        for oy in (-1, 0, 1):
            for ox in (-1, 0, 1):
                k = key[who] + oy * nx + ox
                m = count[k]
                a = torch.repeat_interleave(who, m)
                first = torch.cumsum(m, 0) - m
                b = order[torch.arange(a.numel(), device=x.device) - torch.repeat_interleave(first - start[k], m)]
                dx, dy = x[a] - x[b], y[a] - y[b]
                ok = (torch.sqrt(dx * dx + dy * dy) <= radius) & (a != b) & keep(a, b)
                pa.append(a[ok])
                pb.append(b[ok])
        return torch.cat(pa), torch.cat(pb)


def _limiter(di, dj, dij):
    """MUSCL_Limiter: the increments of both sides."""
    s = torch.where(dj > 0, 1.0, -1.0).to(dj.dtype)
    m = torch.clamp(torch.maximum(torch.minimum(1.3 * s * di, s * dj), torch.minimum(s * di, 1.3 * s * dj)), min=0.0)
    big, first = (m > s * 0.5 * dij) & (m > 0), s * di > s * dj
    half, zero = 0.5 * dij, torch.zeros_like(dij)
    return (torch.where(big, torch.where(first, half, zero), s * m),
            torch.where(big, torch.where(first, zero, half), s * m))


class _Model:
    """The time step on lists of tensors; state = (x, y, u, v, rho) of the host particles."""

    def __init__(self, c, ity, lab, device):
        self.k, self.cfg = _Consts(c.cfg), c.cfg
        self.ms = c.cfg.integrator == S.INTEGRATOR_EULER_PC
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=device)  # noqa: E731
        n = self.n = c.n
        self.state0 = [t(a) for a in (c.pos[:n], c.pos[n:], c.vel[:n], c.vel[n:], c.rho)]
        self.mass, self.type = t(c.mass), t(c.type)
        self.nu = torch.tensor(c.cfg.nu, dtype=torch.float64, device=device)
        self.ity = None if ity is None else t(ity)
        self.lab = None if lab is None else t(lab)
        self.time = 0.0

    def images(self, s):
        """Wrap into the box, append the images (left/right, then bottom/top); returns
        (state, index of each particle's source, types)."""
        c = self.cfg
        out = list(s)
        src = torch.arange(self.n, device=s[0].device)
        if not c.periodic:
            return out, src, self.type
        for ax in (0, 1):
            lo, hi = c.box_lo[ax], c.box_hi[ax]
            p = out[ax]
            out[ax] = torch.where(p > hi, p - (hi - lo), torch.where(p < lo, p + (hi - lo), p))
        band = c.kernel_scale * c.h
        for ax in (0, 1):
            lo, hi = c.box_lo[ax], c.box_hi[ax]
            p = out[ax].detach()
            both = torch.stack([(p <= lo + band) & (p >= lo), (p >= hi - band) & (p <= hi)], 1)
            i, side = torch.nonzero(both, as_tuple=True)
            new = [a[i] for a in out]
            new[ax] = new[ax] + (1 - 2 * side) * (hi - lo)
            out = [torch.cat([a, b]) for a, b in zip(out, new)]
            src = torch.cat([src, src[i]])
        typ = self.type[src].clone()
        typ[self.n:] = S.TYPE_PERIODIC
        return out, src, typ

    def keep(self, typ):
        if self.cfg.pair_rule == S.PAIRS_ONE_FLUID:
            return lambda a, b: (typ[a] == S.TYPE_WATER) | (typ[b] == S.TYPE_WATER)
        return lambda a, b: ~((typ[a] == typ[b]) & (typ[a] == S.TYPE_FIX_GHOST))

    def assign_ghosts(self, s, mass, p, cs, body):
        """Shepard interpolation of the ghosts; returns state, mass, p, c with the ghosts set."""
        k, c = self.k, self.cfg
        x, y, u, v, rho = s
        ghosts = torch.nonzero(self.type == S.TYPE_FIX_GHOST)[:, 0]
        a, b = _near(x, y, c.kernel_scale * k.ghost_h,
                     lambda a, b: (self.type[b] != S.TYPE_FIX_GHOST), targets=ghosts)
        dx, dy = x[a] - x[b], y[a] - y[b]
        w, _ = k.kernel(torch.sqrt(dx * dx + dy * dy), k.ghost_h)
        w = w * mass[b] / rho[b]
        put = lambda t: torch.zeros_like(rho).index_add(0, a, t)  # noqa: E731
        is_body = self.ity == S.TYPE_BODY
        ax, ay = torch.where(is_body, body[2], 0.0), torch.where(is_body, body[3], 0.0)
        sw = put(w)
        ok = (self.type == S.TYPE_FIX_GHOST) & (put(torch.ones_like(w)) >= 3)
        den = torch.where(ok, sw, 1.0)
        pi = put(w * (p[b] + rho[b] * (ax[a] * dx + ay[a] * dy))) / den
        ui, vi, mi = put(w * u[b]) / den, put(w * v[b]) / den, put(w * mass[b]) / den
        lab, early = self.lab, 0.0 < self.time <= c.shock_release_time
        pg = torch.where(is_body | (lab == -6) | (lab == -7), pi, 0.0) if early else pi
        # no-slip walls mirror both components, other labels keep the interpolated velocity
        sign = 1.0 - 2.0 * ((lab == -6) | (lab == -7) | (lab == -8)).to(u.dtype)
        ug, vg = torch.where(is_body, body[0], sign * ui), torch.where(is_body, body[1], sign * vi)
        rg = (pg - c.background_p) / c.c0sq + c.rho0
        g = self.type == S.TYPE_FIX_GHOST
        put_g = lambda old, new, rest: torch.where(ok, new, torch.where(g, rest, old))  # noqa: E731
        cg = math.sqrt(c.c0sq) * (rg / c.rho0) ** 3
        return ([x, y, put_g(u, ug, 0.0), put_g(v, vg, 0.0), put_g(rho, rg, c.rho0)], put_g(mass, mi, 0.0),
                put_g(p, pg, 0.0), put_g(cs, cg, math.sqrt(c.c0sq)))

    def rhs(self, s, typ, mass, body=None, last=False):
        """Rates (drho, ax, ay, avg x, avg y), the shift of a last one, and the body force."""
        k, c = self.k, self.cfg
        p, cs = k.eos(s[4])
        if body is not None:
            s, mass, p, cs = self.assign_ghosts(s, mass, p, cs, body)
        x, y, u, v, rho = s
        a, b = _near(x, y, k.r, self.keep(typ))
        n = rho.numel()
        vol = mass / rho
        put = lambda t: torch.zeros(n, dtype=t.dtype, device=t.device).index_add(0, a, t)  # noqa: E731
        rx, ry = x[a] - x[b], y[a] - y[b]
        d2 = rx * rx + ry * ry
        d = torch.sqrt(d2)
        w, g = k.kernel(d, c.h)
        gx, gy, vb = g * rx, g * ry, vol[b]
        b00, b01, b11 = -put(rx * gx * vb), -put(rx * gy * vb), -put(ry * gy * vb)
        water = typ == S.TYPE_WATER
        if c.renormalize:
            det = torch.where(water, b00 * b11 - b01 * b01, 1.0)
            i00, i01, i11 = (torch.where(water, e / det, f) for e, f in ((b11, 1.0), (-b01, 0.0), (b00, 1.0)))
        else:
            i00, i01, i11 = torch.ones_like(rho), torch.zeros_like(rho), torch.ones_like(rho)

        def grad(phi):
            t = (phi[b] - phi[a]) * vb
            sx, sy = put(t * gx), put(t * gy)
            return i00 * sx + i01 * sy, i01 * sx + i11 * sy

        gr = grad(rho)
        nx, ny = i00[a] * gx + i01[a] * gy, i01[a] * gx + i11[a] * gy
        du, dv, dp = u[a] - u[b], v[a] - v[b], p[a] - p[b]
        ra, rb = rho[a], rho[b]
        rbar, cbar, pbar = 0.5 * (ra + rb), 0.5 * (cs[a] + cs[b]), 0.5 * (p[a] + p[b])
        ex, ey = -rx / d, -ry / d
        sax = say = torch.zeros_like(rho)
        if self.ms or c.xsph_eps:
            f = c.xsph_eps * mass[b] / (ra + rb) * w
            sax, say = -put(f * du), -put(f * dv)
        solver = c.solver
        if solver == S.SOLVER_MS_HLLC_DELTA:
            wx, wy, pstar = self.hllc(a, b, u, v, rho, p, cs, ex, ey)
        else:
            lu = lv = lp = ou = ov = 0.0
            if solver == S.SOLVER_MUSCL_DELTA_SPS:
                sg = torch.where(a < b, 1.0, -1.0).to(rho.dtype)

                def rec(phi, dphi):
                    fx, fy = grad(phi)
                    ga, gb = 0.5 * (fx[a] * rx + fy[a] * ry), 0.5 * (fx[b] * rx + fy[b] * ry)
                    li, lj = _limiter(torch.where(a < b, -ga, gb), torch.where(a < b, gb, -ga), -sg * dphi)
                    return sg * (li + lj), sg * torch.where(a < b, li, lj)

                (lu, ou), (lv, ov), (lp, _) = rec(u, du), rec(v, dv), rec(p, dp)
            wx, wy, pstar = 0.5 * du + ou, 0.5 * dv + ov, pbar
            if solver != S.SOLVER_DELTA_SPS:
                dU = (du + lu) * ex + (dv + lv) * ey
                su = 0.5 * (dp + lp) / (rbar * math.sqrt(math.sqrt(c.c0sq)) ** 2)
                pstar = pbar + 0.5 * torch.minimum(3.0 * torch.clamp(dU, min=0.0), cbar) * rbar * dU
                wx, wy = wx - su * ex, wy - su * ey
        if self.ms:
            wx, wy = wx + sax[a] - sax[b], wy + say[a] - say[b]
        drho = 2.0 * ra * vb * (wx * nx + wy * ny)
        mb, rr = mass[b], 1.0 / (ra * rb)
        vx = du * rx + dv * ry
        phi = c.h * vx / (d2 + (c.fai * c.h) ** 2)
        coef = -2.0 * pstar * rr * mb
        coef = coef - torch.where(vx < 0, mb * (-c.alpha * cbar * phi + c.beta * phi * phi) / rbar, 0.0)
        coef = coef + c.delta_alpha * c.h * cbar * vx / d2 * c.rho0 / ra * vb
        rn = (rx * nx + ry * ny) / d2
        lap = vb * 2.0 * self.nu * rn
        tx, ty = coef * nx + lap * du, coef * ny + lap * dv
        if not self.ms:
            ux, uy = grad(u)
            vx_, vy = grad(v)
            sxy = uy + vx_
            abs2 = 2.0 * (ux * ux + vy * vy) + sxy * sxy
            nut = (k.c012 * k.sps_dl) ** 2 * torch.sqrt(torch.where(water, abs2, 1.0))
            kk, bl = k.c23 * nut * (ux + vy), k.blin * k.sps_dl ** 2 * abs2
            tau = [torch.where(water, e * rho, 0.0)
                   for e in (2.0 * nut * ux - kk - bl, nut * sxy, 2.0 * nut * vy - kk - bl)]
            sxx, sxy, syy = (e[a] + e[b] for e in tau)
            t0 = (sxx * gx + sxy * gy) * rr
            tx = tx + mb * t0
            ty = ty + mb * ((t0 if k.q else 0.0) + syy * gy + sxy * gx) * rr
        sgx, sgy = gr[0][a] + gr[0][b], gr[1][a] + gr[1][b]
        wa = water[a]
        if solver == S.SOLVER_DELTA_SPS:
            f = 2.0 * (rb - ra) / d2
            dif = c.delta * c.h * cbar * ((-f * rx - sgx) * nx + (-f * ry - sgy) * ny) * vb
        else:
            dif = -2.0 * c.delta * c.h * cbar * (rb - ra + 0.5 * (sgx * rx + sgy * ry)) * rn * vb
        drho = put(drho + torch.where(wa, dif, 0.0))
        ax, ay = (torch.where(water, put(t), 0.0) for t in (tx, ty))
        avg = (torch.zeros_like(rho),) * 2 if not self.ms else (sax, say)
        shift = force = None
        if last and c.shifting:
            wdx, _ = k.kernel(torch.tensor(c.dx, dtype=torch.float64, device=d.device), c.h)
            f = -c.shift_beta * c.h * c.h * (1.0 + c.shift_R * (w / wdx) ** 4) * vb
            sx, sy = put(f * nx), put(f * ny)
            amp = torch.sqrt(torch.where(water, sx * sx + sy * sy, 1.0) + 1e-300)
            cap = torch.where(amp > c.shift_max, c.shift_max / amp, 1.0)
            shift = [torch.where(water, e * cap, 0.0) for e in (sx, sy)]
            shift.append(gr[0] * shift[0] + gr[1] * shift[1])
        if last and self.ity is not None:
            m = self.ity[b] == S.TYPE_BODY
            aa, bb = a[m], b[m]
            fp = vol[aa] * -vol[bb] * (p[aa] + p[bb])
            fv = vol[aa] * rho[aa] * vol[bb] * 2.0 * self.nu * rn[m]
            parts = [(fp * nx[m]).sum(), (fp * ny[m]).sum(), (fv * du[m]).sum(), (fv * dv[m]).sum()]
            force = torch.stack(parts + [parts[0] + parts[2], parts[1] + parts[3]])
        return (drho, ax, ay) + avg, shift, force, s, mass, gr, water

    def hllc(self, a, b, u, v, rho, p, cs, ex, ey):
        """v_a - v*, P* of the HLLC state, formed in the frame of the lower id."""
        c = self.cfg
        low = a < b
        i, j = torch.where(low, a, b), torch.where(low, b, a)
        e0, e1 = torch.where(low, ex, -ex), torch.where(low, ey, -ey)
        VL0, VL1, VR0, VR1 = e0 * u[i] + e1 * v[i], -e1 * u[i] + e0 * v[i], e0 * u[j] + e1 * v[j], -e1 * u[j] + e0 * v[j]
        V0 = 0.5 * (VL0 + VR0)
        rL, rR, cL, cR, pL, pR = rho[i], rho[j], cs[i], cs[j], p[i], p[j]
        CL, CR = rL * cL, rR * cR
        us = (VR0 * CL + VL0 * CR + pL - pR) / (CL + CR)
        ps = (pR * CL + pL * CR - CL * CR * (VR0 - VL0)) / (CL + CR)
        rs = (ps - c.background_p) / c.c0sq + c.rho0

        def factor(pk, rk, ck):
            on = (ps > pk) & (rk > rs)
            arg = torch.where(on, (rs / rk) * (ps - pk) / torch.where(on, rk - rs, 1.0), 1.0)
            return torch.where(on, torch.sqrt(arg) / ck, 1.0)

        SL, SR = VL0 - cL * factor(pL, rL, cL), VR0 + cR * factor(pR, rR, cR)
        c1, c2, c3 = SL > V0, (us >= V0) & (V0 >= SL), (SR >= V0) & (V0 >= us)
        pick = lambda q1, q2, q3, q4: torch.where(c1, q1, torch.where(c2, q2, torch.where(c3, q3, q4)))  # noqa: E731
        rH = pick(rL, rL * (SL - VL0) / (SL - us), rR * (SR - VR0) / (SR - us), rR)
        V1, T1 = pick(VL0, us, us, VR0), pick(VL1, VL1, VR1, VR1)
        return u[a] - (e0 * V1 - e1 * T1), v[a] - (e1 * V1 + e0 * T1), c.c0sq * (rH - c.rho0) + c.background_p

    def step(self, s, mass, carried, dt, body=None):
        """One time step; returns (state, mass, rates kept, body force)."""
        c = self.cfg
        force = None
        if self.ms:
            moved = self.ity == S.TYPE_BODY
            s = [torch.where(moved, s[0] + body[0] * dt, s[0]), torch.where(moved, s[1] + body[1] * dt, s[1])] + s[2:]
            water = self.type == S.TYPE_WATER
            first = carried is None
            if first:
                carried, _, _, s, mass, _, _ = self.rhs(s, self.type, mass, body)
            x, y, u, v, rho = s
            dr, ax, ay, gx, gy = carried
            new = [x + dt * (u + gx) + 0.5 * ax * dt * dt, y + dt * (v + gy) + 0.5 * ay * dt * dt, u + dt * ax,
                   v + dt * ay, rho + dr * dt]
            pred = [torch.where(water, e, f) for e, f in zip(new, s)]
            rates, shift, force, pred, mass, _, _ = self.rhs(pred, self.type, mass, body, True)
            d2, ax2, ay2, gx2, gy2 = rates
            new = [x + 0.5 * dt * (pred[2] + u) + gx2 * dt + 0.5 * ax2 * dt * dt,
                   y + 0.5 * dt * (pred[3] + v) + gy2 * dt + 0.5 * ay2 * dt * dt, u + 0.5 * dt * (ax2 + ax),
                   v + 0.5 * dt * (ay2 + ay), rho + 0.5 * (d2 + dr) * dt]
            if shift is not None:
                new[0], new[1], new[4] = new[0] + shift[0], new[1] + shift[1], new[4] + shift[2]
            return [torch.where(water, e, f) for e, f in zip(new, pred)], mass, rates, force
        n = self.n
        full, src, typ = self.images(s)
        m = mass[src]
        host = full[4].new_ones(full[4].numel(), dtype=torch.bool)
        host[n:] = False
        pad = lambda r: [torch.cat([e[:n], torch.zeros_like(full[4][n:])]) for e in r]  # noqa: E731
        rates = self.rhs(full, typ, m)[0] if carried is None else pad(carried)
        x, y, u, v, rho = full
        sums = None
        for stage in range(4):
            dr, ax, ay, gx, gy = pad(rates)
            if stage == 3:
                new_u = u + (sums[1] + ax) * dt / 6.0 + gx
                new_v = v + (sums[2] + ay) * dt / 6.0 + gy
                new = [x + (sums[3] + new_u) * dt / 6.0 + 0.5 * dt * dt * ax,
                       y + (sums[4] + new_v) * dt / 6.0 + 0.5 * dt * dt * ay, new_u, new_v,
                       rho + (sums[0] + dr) * dt / 6.0]
                break
            f = 0.5 * dt if stage < 2 else dt
            nu_, nv_ = u + f * ax + gx, v + f * ay + gy
            cur = [torch.where(host, e, o) for e, o in zip([x + f * nu_, y + f * nv_, nu_, nv_, rho + dr * f], full)]
            add = [dr, ax, ay, nu_, nv_]
            sums = add if stage == 0 else [e + 2.0 * o for e, o in zip(sums, add)]
            rates, shift, _, _, _, _, _ = self.rhs(cur, typ, m, last=stage == 2)
        if shift is not None and not self.reinit_now:
            new[0], new[1], new[4] = new[0] + shift[0], new[1] + shift[1], new[4] + shift[2]
        new = [torch.where(host, e, o) for e, o in zip(new, full)]
        if self.reinit_now:
            new[4] = self.mls(new, typ, m)
            if shift is not None:
                new[0], new[1], new[4] = new[0] + shift[0], new[1] + shift[1], new[4] + shift[2]
        return [e[:n] for e in new], mass, [e[:n] for e in rates], None

    reinit_now = False

    def mls(self, s, typ, mass):
        """Moving-least-squares density of the water particles (order 6 or 3)."""
        k, c = self.k, self.cfg
        x, y, _, _, rho = s
        a, b = _near(x, y, k.r, self.keep(typ))
        dx, dy = (x[b] - x[a]) / c.h, (y[b] - y[a]) / c.h
        w, _ = k.kernel(torch.sqrt((x[a] - x[b]) ** 2 + (y[a] - y[b]) ** 2), c.h)
        q = [torch.ones_like(dx), dx, dy] + ([dx * dx, dx * dy, dy * dy] if c.mls_order == 6 else [])
        m, n = len(q), rho.numel()
        A = torch.zeros(n, m, m, dtype=rho.dtype, device=rho.device)
        r = torch.zeros(n, m, dtype=rho.dtype, device=rho.device)
        for i in range(m):
            r[:, i].index_add_(0, a, w * rho[b] * q[i])
            for j in range(m):
                A[:, i, j].index_add_(0, a, w * q[i] * q[j])
        host = torch.arange(n, device=rho.device) < self.n
        eye = torch.eye(m, dtype=rho.dtype, device=rho.device)
        A = torch.where(host[:, None, None], A + c.mls_alpha ** 3 * eye, eye)
        one = torch.zeros(n, m, dtype=rho.dtype, device=rho.device)
        one[:, 0] = 1.0
        return torch.where(host & (typ == S.TYPE_WATER), (torch.linalg.solve(A, one) * r).sum(1), rho)


def _cat(x, y):
    return torch.cat([x, y])


def exact(case, seed):
    c, ity, lab, target = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m = _Model(c, ity, lab, dev)
    n, kind, dt = c.n, case["kind"], _dt(c.cfg)
    flat = lambda t: t.detach().cpu().numpy()  # noqa: E731
    body = torch.tensor([1.0, 0.0, 0.0, 0.0], dtype=torch.float64, device=dev) if m.ms else None
    if kind == "pairs":
        s, src, typ = m.images(m.state0)
        a, b = _near(s[0], s[1], m.k.r, m.keep(typ))
        a, b = a[a < b], b[a < b]
        o = torch.argsort(a * s[0].numel() + b)
        a, b = a[o], b[o]
        rx, ry = s[0][a] - s[0][b], s[1][a] - s[1][b]
        w, g = m.k.kernel(torch.sqrt(rx * rx + ry * ry), c.cfg.h)
        pad = lambda t: flat(torch.nn.functional.pad(t, (0, _pair_cap(c) - t.numel())))  # noqa: E731
        return {"pair_i": pad((a + 1).int()), "pair_j": pad((b + 1).int()), "pair_number": int(a.numel()),
                "w": pad(w), "dwdx": np.concatenate([pad(g * rx), pad(g * ry)])}
    if kind == "rhs":
        with torch.no_grad():
            s, src, typ = m.images(m.state0)
            (dr, ax, ay, gx, gy) = [e[:n] for e in m.rhs(s, typ, m.mass[src])[0]]
        return {"drhodt": flat(dr), "acc": flat(_cat(ax, ay)), "avg_vel": None, "fs": None, "near": None}
    if kind in ("run", "coupled"):
        steps = case.get("steps", 1)
        with torch.no_grad():
            s, mass, rates, force = m.state0, m.mass, None, None
            for k in range(steps):
                m.time += dt
                m.reinit_now = bool(c.cfg.mls_order) and (k + 1) % c.cfg.mls_every == 0
                s, mass, rates, force = m.step(s, mass, rates, dt, body)
            water = m.type == S.TYPE_WATER
            ke = float((0.5 * mass * (s[2] ** 2 + s[3] ** 2))[water].sum())
        out = {"pos": flat(_cat(s[0], s[1])), "vel": flat(_cat(s[2], s[3])), "rho": flat(s[4])}
        if kind == "run":
            out["kinetic_energy"] = ke
            if m.ms:
                out["body_force"] = flat(force)
        return out
    # adjoint: reverse-mode differentiation of the same step, recomputed step by step
    s = [e.clone().requires_grad_(True) for e in m.state0]
    start, mass, rates = s, m.mass, None
    m.nu.requires_grad_(True)
    steps = case["steps"]
    motion = body.repeat(steps, 1).requires_grad_(True) if m.ms else None
    drag = torch.zeros((), dtype=torch.float64, device=dev)

    def one(first, now, *flat_in):
        m.time = now
        st, ms_, rt = list(flat_in[:5]), flat_in[5], None if first else list(flat_in[6:11])
        st, ms_, rt, f = m.step(st, ms_, rt, dt, flat_in[-1] if m.ms else None)
        return tuple(st) + (ms_,) + tuple(rt) + ((f,) if m.ms else ())

    for k in range(steps):
        args = tuple(s) + (mass,) + tuple(rates if rates is not None else s)
        got = checkpoint(one, k == 0, (k + 1) * dt, *args, *((motion[k],) if m.ms else ()), use_reentrant=False)
        s, mass, rates = list(got[:5]), got[5], list(got[6:11])
        if m.ms:
            drag = drag + dt * got[11][4]
    if m.ms:
        loss = drag
    else:
        tg = torch.as_tensor(target, device=dev)
        loss = ((_cat(s[2], s[3]) - tg) ** 2).sum()
    loss.backward()
    zero = lambda t: torch.zeros_like(t) if t.grad is None else t.grad  # noqa: E731
    x, y, u, v, rho = (zero(e) for e in start)
    out = {"vel0": flat(_cat(u, v)), "rho0": flat(rho), "pos0": flat(_cat(x, y)), "nu": float(m.nu.grad),
           "loss": float(loss.detach())}
    if m.ms:
        out["motion"] = flat(motion.grad)
    return out
