"""sph_init that fails (a capacity whose arrays do not fit the GPU) gives an error code,
no handle, and the device memory back; the next handle works."""
import ctypes

import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu


def test_failed_init_gives_everything_back(lib):
    import torch
    case = S.make_tgv(24)
    with S.Simulation(case.cfg, case.n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
    free, _ = torch.cuda.mem_get_info()
    for _ in range(3):
        h = ctypes.c_void_p(1)
        assert lib.sph_init(ctypes.byref(case.cfg), 400_000_000, ctypes.byref(h)) == -5     # SPH_E_CUDA
        assert not h.value
    assert torch.cuda.mem_get_info()[0] == free
    with S.Simulation(case.cfg, case.n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        sim.time_iteration(2, S.baseline_dt(case.cfg))
