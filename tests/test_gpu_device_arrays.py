"""Callers whose arrays already are in device memory: the state goes in and out through
sph_update_state and sph_get_state as with host arrays."""
import ctypes

import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [47, 500])
def test_state_round_trip_in_device_arrays(lib, side):
    import torch
    case = S.make_tgv(side, jitter=0.1, seed=side)
    n = case.n
    rng = np.random.default_rng(side)
    want = [rng.random(2 * n), rng.standard_normal(2 * n), 1.0 + 1e-3 * rng.random(n)]
    into = [torch.from_numpy(a).cuda() for a in want]
    out = [torch.zeros(m * n, dtype=torch.float64, device="cuda") for m in (2, 2, 1)]
    torch.cuda.synchronize()
    p = lambda t: ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))
    with S.Simulation(case.cfg, n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        assert lib.sph_update_state(sim.h, n, *[p(t) for t in into]) == 0
        assert lib.sph_get_state(sim.h, n, *[p(t) for t in out], None) == 0
    for a, b in zip(out, want):
        assert np.array_equal(a.cpu().numpy(), b)
