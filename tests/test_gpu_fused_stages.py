"""The stages applied inside the gather and the force kernels, in the driver and
solver combinations that take different routes: the Taylor-Green solvers with the
Euler predictor-corrector, a moving-square solver with Runge-Kutta, shifting on
and off, a density re-initialisation between fused steps; against the oracle in
FP64 (1e-10 norm-wise, as the parity tests) and mixed against FP64."""
import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


def _case(kind, integrator, shifting, precision=S.PREC_FP64):
    if kind == "ms":
        case, _ = S.make_moving_square(dx=0.1, solver=S.SOLVER_MS_MODLR_DELTA, precision=precision, jitter=0.05, seed=2)
        case.cfg.mls_order = 0
    else:
        solver = {"muscl": S.SOLVER_MUSCL_DELTA_SPS, "plain": S.SOLVER_DELTA_SPS, "mls": S.SOLVER_MODLR_DELTA_SPS}[kind]
        case = S.make_tgv(33, solver=solver, precision=precision, jitter=0.1, seed=6)
        if kind == "mls":
            case.cfg.mls_order, case.cfg.mls_every, case.cfg.mls_alpha = 3, 3, 1e-4
    case.cfg.integrator = integrator
    case.cfg.shifting = shifting
    return case


ROUTES = [(k, i, s) for k in ("muscl", "plain", "mls", "ms") for i in (S.INTEGRATOR_RK4_REUSE, S.INTEGRATOR_EULER_PC)
          for s in (0, 1)]


def _run(case, dt, chunks):
    with S.Simulation(case.cfg, case.n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        for c in chunks:
            sim.time_iteration(c, dt)
        return sim.get_state()


@pytest.mark.parametrize("kind,integrator,shifting", ROUTES)
def test_steps_match_the_oracle(lib, oracle, kind, integrator, shifting):
    case = _case(kind, integrator, shifting)
    dt = 0.2 * case.cfg.h / np.sqrt(case.cfg.c0sq)
    ref = oracle.OracleSim(case.cfg, case.pos, case.vel, case.rho, case.mass, case.type)
    ref.run(5, dt)
    rpos, rvel, rrho, _ = ref.state()
    one = _run(case, dt, [5])
    assert np.abs(one[0] - rpos).max() < 1e-12
    assert relerr(one[1], rvel) < 1e-10
    assert relerr(one[2], rrho) < 1e-10
    # state reads between the steps change nothing
    for a, b in zip(one, _run(case, dt, [1, 2, 1, 1])):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kind,integrator,shifting", [r for r in ROUTES if r[0] != "mls"])
def test_mixed_steps_follow_fp64(lib, kind, integrator, shifting):
    dt = None
    out = []
    for prec in (S.PREC_FP64, S.PREC_MIXED):
        case = _case(kind, integrator, shifting, prec)
        dt = 0.2 * case.cfg.h / np.sqrt(case.cfg.c0sq)
        out.append(_run(case, dt, [5]))
    (p, v, r, _), (pm, vm, rm, _) = out
    assert np.linalg.norm(vm - v) <= 1e-5 * np.linalg.norm(v)      # the mixed path's bound
    assert np.abs(pm - p).max() <= 1e-5 * dt * 5 * np.abs(v).max() + 1e-8
