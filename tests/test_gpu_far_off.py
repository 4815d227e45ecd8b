"""A particle far off the cell grid: a coordinate whose cell number does not fit an int
(or is no number at all), with the other coordinate on the grid, so that the list
builders scan the rows beside it.  The step and the pair search report SPH_E_DOMAIN,
for particle counts on both list builders, and the handle takes a clean state after."""
import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu

E_DOMAIN = -8


def _code(fn, *args):
    try:
        fn(*args)
    except S.SphError as e:
        return e.code
    return 0


@pytest.mark.parametrize("side", [32, 260])        # 8 lanes per particle, a thread per particle
@pytest.mark.parametrize("precision", [S.PREC_FP64, S.PREC_MIXED])
@pytest.mark.parametrize("axis", [0, 1])
def test_far_off_coordinate_is_reported(lib, side, precision, axis):
    case = S.make_tgv(side, precision=precision, jitter=0.1, seed=side)
    dt = S.baseline_dt(case.cfg)
    with S.Simulation(case.cfg, case.n) as sim:
        for x in (np.inf, -np.inf, 1e300, -1e300, 1e12, -1e12, np.nan):
            pos = case.pos.copy()
            pos[axis * case.n + case.n // 2] = x
            sim.set_state(pos, case.vel, case.rho, case.mass, case.type)
            assert _code(sim.time_iteration, 1, dt) == E_DOMAIN
            sim.set_state(pos, case.vel, case.rho, case.mass, case.type)
            assert _code(sim.find_particle_pair, 20 * case.n) == E_DOMAIN
        # thrown out along the axis by the first of two steps
        vel = case.vel.copy()
        vel[axis * case.n + case.n // 2] = 1e15 / dt
        sim.set_state(case.pos, vel, case.rho, case.mass, case.type)
        assert _code(sim.time_iteration, 2, dt) == E_DOMAIN
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        d = sim.time_iteration(2, dt)
        assert np.isfinite(d.kinetic_energy) and d.kinetic_energy > 0.0
