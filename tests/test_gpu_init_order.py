"""The clears of a new handle are ordered before its work, whatever the caller has queued
on the default stream: the surface marks of the first right-hand side and the wall
labels are still there once that work has run."""
import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [S.PREC_FP64, S.PREC_MIXED])
def test_clears_do_not_wait_for_the_default_stream(lib, precision):
    import torch
    case = S.make_tgv(40, solver=S.SOLVER_MODLR_DELTA_SPS, precision=precision, jitter=0.05, seed=7)
    case.cfg.periodic = 0                   # an open block of fluid: its rim is a free surface
    case.cfg.free_surface = 1
    n = case.n
    labels = np.arange(n, dtype=np.int32) % 5
    busy = torch.ones(8192, 8192, dtype=torch.bfloat16, device="cuda")

    def run(sim):
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        sim.set_boundary_labels(labels)
        return int(sim.single_step_compute()["fs"].sum())

    with S.Simulation(case.cfg, n) as sim:  # (kernels loaded)
        want = run(sim)
    assert want > 0
    for _ in range(5):                      # (a handle's start may take long on a busy host)
        for _ in range(300):
            busy @ busy
        done = torch.cuda.Event()
        done.record()
        with S.Simulation(case.cfg, n) as sim:
            got = run(sim)
            early = not done.query()        # the default stream is still at work
            torch.cuda.synchronize()
            assert got == want
            assert sim.diagnostics().n_surface == want
            image = sim.restart_save()
            at = 64 + (2 * 16 + 3 * 8 + 2 * 4) * n
            assert np.array_equal(np.frombuffer(image, np.int32, n, at), labels)
        if early:
            return
    pytest.fail("the queued work always ended too soon for the test to mean anything")
