"""Whole steps of a block of fluid with open edges: the surface test at the end of pass
A, the near-surface marks in pass C and the shift that skips the marked particles, at
particle counts on every lane count of the FP64 loops; against the oracle in FP64
(1e-10 norm-wise, as the parity tests) and mixed against FP64 (1e-5, the mixed path's
bound)."""
import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


def _case(kind, side, precision=S.PREC_FP64):
    if kind == "ms":
        case, _ = S.make_moving_square(dx=2.0 / side, solver=S.SOLVER_MS_MODLR_DELTA, precision=precision,
                                       jitter=0.05, seed=2)
        case.cfg.mls_order = 0
        keep = (case.type == S.TYPE_WATER) & (case.pos[case.n:] < 1.2)      # a tank with a free surface at y = 1.2
        keep |= case.type != S.TYPE_WATER
        two = np.concatenate([keep, keep])
        case = S.TgvCase(case.cfg, case.pos[two], case.vel[two], case.rho[keep], case.mass[keep], case.type[keep])
    else:
        solver = {"modlr": S.SOLVER_MODLR_DELTA_SPS, "muscl": S.SOLVER_MUSCL_DELTA_SPS}[kind]
        case = S.make_tgv(side, solver=solver, precision=precision, jitter=0.1, seed=side)
        case.cfg.periodic = 0
    case.cfg.free_surface = 1
    case.cfg.shifting = 1
    return case


def _run(case, dt):
    with S.Simulation(case.cfg, case.n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        d = sim.time_iteration(5, dt)
        return sim.get_state(), d.n_surface


ROUTES = [("modlr", 40), ("muscl", 40), ("muscl", 140), ("modlr", 310), ("ms", 40), ("ms", 120)]


@pytest.mark.parametrize("kind,side", ROUTES)
def test_steps_with_a_free_surface_match_the_oracle(lib, oracle, kind, side):
    case = _case(kind, side)
    dt = 0.1 * case.cfg.h / np.sqrt(case.cfg.c0sq)
    ref = oracle.OracleSim(case.cfg, case.pos, case.vel, case.rho, case.mass, case.type)
    ref.run(5, dt)
    rpos, rvel, rrho, _ = ref.state()
    (pos, vel, rho, _), ns = _run(case, dt)
    assert ns > side
    assert np.abs(pos - rpos).max() < 1e-12
    assert relerr(vel, rvel) < 1e-10
    assert relerr(rho, rrho) < 1e-10
    # the marks matter: without them the shift moves the particles at the edge
    case.cfg.free_surface = 0
    (other, _, _, _), _ = _run(case, dt)
    assert np.abs(other - pos).max() > 1e-8


@pytest.mark.parametrize("kind,side", ROUTES)
def test_mixed_steps_with_a_free_surface_follow_fp64(lib, kind, side):
    out = []
    for prec in (S.PREC_FP64, S.PREC_MIXED):
        case = _case(kind, side, prec)
        dt = 0.1 * case.cfg.h / np.sqrt(case.cfg.c0sq)
        out.append(_run(case, dt))
    ((p, v, r, _), ns), ((pm, vm, rm, _), nm) = out
    assert ns > side and nm == ns
    assert np.linalg.norm(vm - v) <= 1e-5 * np.linalg.norm(v)
    assert np.abs(pm - p).max() <= 1e-5 * dt * 5 * np.abs(v).max() + 1e-8
