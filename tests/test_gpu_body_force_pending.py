"""The body force of steps taken without a diagnostics argument stays readable when the
body is changed before it is read: sph_diagnostics then still reports the force of the
last RHS, whether the new body is larger (its buffers are then taken anew), smaller or
empty."""
import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dx", [0.05, 0.0125])
def test_pending_body_force_survives_a_new_body(lib, dx):
    case, ity = S.make_moving_square(dx=dx, jitter=0.05, seed=2)
    dt = 0.25 * case.cfg.h / np.sqrt(case.cfg.c0sq)
    body = np.flatnonzero(ity == S.TYPE_BODY)

    def types(m):
        t = np.zeros_like(ity)
        t[body[:m]] = S.TYPE_BODY
        return t

    sizes = [5, 40, body.size // 2, body.size, 7, 0]
    out = []
    for change in (False, True):
        with S.Simulation(case.cfg, case.n) as sim:
            sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
            got = []
            for k, m in enumerate(sizes[:-1]):
                sim.set_initial_type(types(m))
                assert lib.sph_step(sim.h, 1, dt, None) == 0
                if change:
                    sim.set_initial_type(types(sizes[k + 1]))
                got.append(np.array(sim.diagnostics().body_force[:]))
            out.append(np.array(got))
    assert (np.abs(out[0]).max(axis=1) > 0.0).all()
    assert np.array_equal(out[0], out[1])


def test_setting_a_body_takes_no_device_memory(lib):
    """The buffers of the body force are the handle's from its start, so that no call in
    between can fail half-way for want of memory: a million body particles, free memory
    the same before and after."""
    import torch
    case = S.make_tgv(1000)
    with S.Simulation(case.cfg, case.n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        sim.set_initial_type(case.type)
        before, _ = torch.cuda.mem_get_info()
        sim.set_initial_type(np.full(case.n, S.TYPE_BODY, np.int32))
        after, _ = torch.cuda.mem_get_info()
    assert after == before
