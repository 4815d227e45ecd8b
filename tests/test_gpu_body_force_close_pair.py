"""The body force of a pair closer than 1e-8 h, where the kernel gradient is zero
(compute_kernel): in units in which h is above 10 such a pair passes the pair search's
1e-7.  Against the oracle, FP64."""
import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu


def test_body_force_of_a_coinciding_pair(lib, oracle):
    case, ity = S.make_moving_square(dx=20.0, lx=800.0, ly=400.0, D=200.0, solver=S.SOLVER_MS_MODLR_DELTA,
                                     jitter=0.05, seed=5)
    case.cfg.shifting, case.cfg.mls_order = 0, 0
    n = case.n
    body = np.flatnonzero(ity == S.TYPE_BODY)
    water = np.flatnonzero(case.type == S.TYPE_WATER)
    pos = case.pos.copy()
    # the water particle next to the body moves onto one of the body's
    b = body[0]
    near = water[np.argmin((pos[water] - pos[b]) ** 2 + (pos[n + water] - pos[n + b]) ** 2)]
    pos[near], pos[n + near] = pos[b] + 1.5e-7, pos[n + b]
    d = pos[near] - pos[b]
    assert d >= 1e-7 and d <= 1e-8 * case.cfg.h
    with S.Simulation(case.cfg, n) as sim:
        sim.set_state(pos, case.vel, case.rho, case.mass, case.type)
        sim.set_initial_type(ity)
        sim.single_step_compute()
        got = np.array(sim.diagnostics().body_force[:])
    want = np.array(oracle.rhs_body_force(case.cfg, pos, case.vel, case.rho, case.mass, case.type, ity))
    assert np.abs(got - want).max() <= 1e-10 * np.abs(want).max()
