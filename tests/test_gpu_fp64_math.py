"""The FP64 pair arithmetic that replaces library division and square root:
rcp64 and rsqrt64 (common.cuh) against the correctly rounded 1/x and 1/sqrt(x),
and the support test on the squared distance against the oracle's
sqrt(d2) <= kernel_scale h on lattices whose distances fall on the bound."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def _ulps(a, b):
    return np.abs(a.view(np.int64) - b.view(np.int64))


def test_newton_reciprocals_within_two_ulp(lib, tmp_path):
    """The correction step leaves e^3 < 2^-57 of the 20-bit estimate's error; the
    last multiply-add and the rounding of e add at most about one ulp."""
    import torch
    so = str(tmp_path / "fp64_math.so")
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
                    "-shared", "-o", so, os.path.join(HERE, "fp64_math.cu")], check=True)
    fn = ctypes.CDLL(so).fp64_math
    fn.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 3
    rng = np.random.default_rng(0)
    # every mantissa range, the decades squared distances and densities fall in, and powers of two
    x = np.concatenate([10.0 ** rng.uniform(-16, 8, 1 << 20), 1.0 + rng.random(1 << 18), 2.0 ** np.arange(-60, 60)])
    xd = torch.from_numpy(x).cuda()
    r, q = torch.empty_like(xd), torch.empty_like(xd)
    assert fn(x.size, xd.data_ptr(), r.data_ptr(), q.data_ptr()) == 0
    exact = np.sqrt(x.astype(np.longdouble))
    assert _ulps(r.cpu().numpy(), 1.0 / x).max() <= 2
    assert _ulps(q.cpu().numpy(), (1.0 / exact).astype(np.float64)).max() <= 2


@pytest.mark.parametrize("h_over_dx", [1.0, 1.5, float(np.sqrt(2.0)), float(np.sqrt(5.0)) / 2])
def test_support_bound_on_lattice_ties(lib, oracle, h_over_dx):
    """kernel_scale h equal to lattice distances (2, 3, 2 sqrt 2, sqrt 5 times dx): which
    neighbours on the bound count is decided by rounding, and fra_v (each neighbour
    adds its V) has to decide as the reference's test does."""
    case = S.make_tgv(40)
    case.cfg.h = h_over_dx * case.cfg.dx
    ext = oracle.periodic_images(case.cfg, case.pos, case.vel, case.rho, case.mass, case.type)[:5]
    ref = oracle.rhs(case.cfg, *ext)
    with S.Simulation(case.cfg, case.n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        sim.single_step_compute()
        fra = sim.field(S.FIELD_FRA_V)
    assert np.abs(fra - ref["fra_v"][:case.n]).max() < 1e-12
