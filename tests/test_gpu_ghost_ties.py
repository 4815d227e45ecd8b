"""The ghost assignment's radius on lattice ties: neighbours at exactly the distance the
radius rounds to (sqrt(13), sqrt(18), sqrt(10) spacings, a spacing that is a power of
two, so that all distances are exact) count as in the reference's sqrt(d2) <= radius,
whose square may round below d2.  A Gaussian at kernel_scale 2 has weight there.  One
step against the oracle, FP64, 1e-10 norm-wise as the other ghost tests."""
import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("k", [10, 13, 18])
def test_ghosts_count_neighbours_on_the_radius(lib, oracle, k):
    dx = 0.125
    case, ity = S.make_moving_square(dx=dx, solver=S.SOLVER_MS_MODLR_DELTA)
    cfg = case.cfg
    cfg.kernel_model = S.KERNEL_GAUSSIAN
    cfg.kernel_scale = 2.0
    cfg.ghost_h_factor = 2.0
    cfg.h = float(np.sqrt(float(k))) * dx / 4.0          # kernel_scale * 2 h = sqrt(k) dx, exactly
    cfg.shifting, cfg.mls_order, cfg.ghost_assign = 0, 0, 1
    assert cfg.kernel_scale * (cfg.ghost_h_factor * cfg.h) == np.sqrt(float(k)) * dx
    lab = S.moving_square_labels(case, ity)
    rng = np.random.default_rng(k)
    water = case.type == S.TYPE_WATER
    vel, rho = case.vel.copy(), case.rho.copy()
    vel[:case.n][water] = rng.uniform(-0.5, 0.5, water.sum())
    vel[case.n:][water] = rng.uniform(-0.5, 0.5, water.sum())
    rho[water] *= 1.0 + 1e-3 * rng.uniform(-1.0, 1.0, water.sum())
    dt = 0.1 * cfg.h / np.sqrt(cfg.c0sq)
    oracle.set_ghost_state(lab, (0.0, 0.0), (0.0, 0.0), 20.0)
    ref = oracle.OracleSim(cfg, case.pos, vel, rho, case.mass, case.type)
    ref.set_initial_type(ity)
    ref.run(1, dt)
    rpos, rvel, rrho, _ = ref.state()
    with S.Simulation(cfg, case.n) as sim:
        sim.set_state(case.pos, vel, rho, case.mass, case.type)
        sim.set_initial_type(ity)
        sim.set_boundary_labels(lab)
        sim.set_body_motion((0.0, 0.0))
        sim.set_time(20.0)
        sim.time_iteration(1, dt)
        pos, gvel, grho, _ = sim.get_state()
    assert relerr(gvel, rvel) < 1e-10
    assert relerr(grho - cfg.rho0, rrho - cfg.rho0) < 1e-10
    assert np.abs(pos - rpos).max() < 1e-12
