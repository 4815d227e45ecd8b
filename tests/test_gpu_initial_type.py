"""sph_set_initial_type is complete on return: a page-locked array that the caller
refills at once leaves the handle with the values it was called with, also when no
particle belongs to the body."""
import struct

import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [47, 700])
def test_page_locked_initial_types_without_a_body(lib, side):
    import torch
    case = S.make_tgv(side, jitter=0.1, seed=1)
    n = case.n
    want = (np.arange(n, dtype=np.int32) % 3) + 1          # no SPH_TYPE_BODY among them
    assert not (want == S.TYPE_BODY).any()
    ity = torch.zeros(n, dtype=torch.int32).pin_memory().numpy()
    busy = torch.ones(8192, 8192, dtype=torch.bfloat16, device="cuda")
    with S.Simulation(case.cfg, n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        for _ in range(8):
            ity[:] = want
            # the copy waits in the handle's stream, behind a kernel that finds the GPU busy
            sim.single_step_compute()
            for _ in range(10):
                busy @ busy
            sim.set_initial_type(ity)
            ity[:] = 77
            image = sim.restart_save()
            n_saved, = struct.unpack_from("<i", image, 12)
            assert n_saved == n
            at = 64 + (2 * 16 + 3 * 8 + 4) * n             # header, x, v, rho, m, SPS m, type
            got = np.frombuffer(image, np.int32, n, at)
            assert np.array_equal(got, want)
