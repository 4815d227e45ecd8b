"""Copies between the handle and the caller's arrays: sizes below one page-locked
chunk (1 MiB), around it, and enough for the threads that share larger copies;
pageable and page-locked arrays; arrays the caller leaves out."""
import ctypes

import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu


def _p(a):
    return None if a is None else a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


@pytest.mark.parametrize("side", [3, 47, 161, 162, 256, 363, 700])
@pytest.mark.parametrize("locked", [False, True])
def test_state_round_trip(lib, side, locked):
    import torch
    case = S.make_tgv(side, jitter=0.1, seed=side)
    n = case.n
    rng = np.random.default_rng(side)
    with S.Simulation(case.cfg, n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        for _ in range(2):                       # the second time the chunks are reused
            pos, vel, rho = rng.random(2 * n), rng.standard_normal(2 * n), 1.0 + 1e-3 * rng.random(n)
            if locked:
                pos, vel, rho = (torch.from_numpy(a).pin_memory().numpy() for a in (pos, vel, rho))
            sim.update_state(pos, vel, rho)
            keep = [a.copy() for a in (pos, vel, rho)]
            pos[:], vel[:], rho[:] = 0.0, 0.0, 1.0      # the caller refills its arrays at once
            out = [np.full(m * n, -1.0) for m in (2, 2, 1, 1)]
            if locked:
                out = [torch.from_numpy(a).pin_memory().numpy() for a in out]
            assert lib.sph_get_state(sim.h, n, *[_p(a) for a in out]) == 0
            for a, b in zip(out, keep):
                assert np.array_equal(a, b)
            only = np.full(n, -1.0)
            assert lib.sph_get_state(sim.h, n, None, None, _p(only), None) == 0
            assert np.array_equal(only, keep[2])


def test_pair_arrays_short_of_the_count(lib):
    """A capacity below the count fills the prefix of every array, dwdx's second block at
    the capacity's offset, and leaves out what the caller leaves out."""
    case = S.make_tgv(120, jitter=0.1, seed=8)
    with S.Simulation(case.cfg, case.n) as sim:
        sim.set_state(case.pos, case.vel, case.rho, case.mass, case.type)
        full = sim.find_particle_pair(12 * case.n)
        m = full["pair_number"]
        for cap in (1, 1000, m - 1, m, m + 5):
            pi, pj = np.zeros(cap, np.int32), np.zeros(cap, np.int32)
            w, dw = np.zeros(cap), np.zeros(2 * cap)
            cnt = ctypes.c_longlong(0)
            ip = ctypes.POINTER(ctypes.c_int)
            rc = lib.sph_find_particle_pair(sim.h, cap, pi.ctypes.data_as(ip), pj.ctypes.data_as(ip), _p(w), _p(dw),
                                            ctypes.byref(cnt))
            assert rc == (0 if cap >= m else -2) and cnt.value == m
            k = min(cap, m)
            assert np.array_equal(pi[:k], full["pair_i"][:k]) and np.array_equal(pj[:k], full["pair_j"][:k])
            assert np.array_equal(w[:k], full["w"][:k])
            assert np.array_equal(dw[:k], full["dwdx"][0][:k]) and np.array_equal(dw[cap:cap + k], full["dwdx"][1][:k])
            pi[:] = 0
            rc = lib.sph_find_particle_pair(sim.h, cap, pi.ctypes.data_as(ip), pj.ctypes.data_as(ip), None, None,
                                            ctypes.byref(cnt))
            assert np.array_equal(pi[:k], full["pair_i"][:k])
