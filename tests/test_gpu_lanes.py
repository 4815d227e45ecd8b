"""One right-hand side against the oracle at particle counts (host + images) on both
sides of the sizes where the FP64 loops and the list build change their lanes per
particle: passes A and C 4 lanes below 17,000, pass A 2 below 60,000, pass C 2
below 90,000, lists 8 below 60,000.  1e-10 norm-wise, as the parity tests."""
import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("side", [24, 124, 126, 234, 238, 239, 294, 297])
@pytest.mark.parametrize("solver", [S.SOLVER_MUSCL_DELTA_SPS, S.SOLVER_DELTA_SPS])
def test_rhs_across_lane_counts(lib, oracle, side, solver):
    case = S.make_tgv(side, solver=solver, jitter=0.1, seed=side)
    ext = oracle.periodic_images(case.cfg, case.pos, case.vel, case.rho, case.mass, case.type)[:5]
    ref = oracle.rhs(case.cfg, *ext)
    n, m = case.n, ext[2].size
    with S.Simulation(case.cfg, n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        got = sim.single_step_compute()
        fra, tau = sim.field(S.FIELD_FRA_V), sim.field(S.FIELD_TAU)
    assert relerr(got["drhodt"], ref["drhodt"][:n]) < 1e-10
    assert relerr(got["acc"], np.concatenate([ref["acc"][:n], ref["acc"][m:m + n]])) < 1e-10
    assert relerr(fra, ref["fra_v"][:n]) < 1e-12
    assert relerr(tau[:n], ref["tau"][:n]) < 1e-10


@pytest.mark.parametrize("dx", [0.1, 0.02, 0.0125])
def test_moving_square_rhs_across_lane_counts(lib, oracle, dx):
    """About 1,300, 21,500 and 54,000 particles, Gaussian support (45 list entries, past the
    32 that the thread-per-particle list build stages)."""
    case, ity = S.make_moving_square(dx=dx, solver=S.SOLVER_MS_MODLR_DELTA, jitter=0.05, seed=7)
    ref = oracle.rhs(case.cfg, case.pos, case.vel, case.rho, case.mass, case.type)
    with S.Simulation(case.cfg, case.n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        sim.set_initial_type(ity)
        got = sim.single_step_compute()
    water = case.type == S.TYPE_WATER
    assert relerr(got["drhodt"][water], ref["drhodt"][water]) < 1e-10
    assert relerr(got["acc"], ref["acc"]) < 1e-10


def test_phase_times_cover_the_steps(lib):
    """The phases, stamped by the kernels, add up to the events around the steps, and a
    pause of the host between two calls is in neither."""
    import time
    case = S.make_tgv(300, jitter=0.1, seed=1)
    dt = S.baseline_dt(case.cfg)
    with S.Simulation(case.cfg, case.n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        sim.time_iteration(2, dt)
        sim.reset_timings()
        sim.time_iteration(5, dt)
        time.sleep(0.2)
        sim.time_iteration(5, dt)
        t = sim.timings()
    phases = t.sort_ms + t.pass_a_ms + t.surface_ms + t.pass_c_ms + t.update_ms + t.images_ms
    assert t.steps == 10 and t.pass_a_ms > 0 and t.pass_c_ms > 0 and t.sort_ms > 0 and t.images_ms > 0
    assert 0.8 * t.total_ms < phases < 1.05 * t.total_ms
    assert t.total_ms < 100.0
