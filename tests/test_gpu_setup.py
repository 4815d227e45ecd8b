"""The step set-up (image numbering, counting sort into cells, neighbour lists)
through find_particle_pair against the oracle: particle counts around the image
block (1024 host particles), boxes thinner than two image bands (a particle then
has images on both sides of an axis), particles that are not binned, and cells
whose population is far from the lattice's.  Pairs are compared as the emitted
list, so ids, numbering and order all count."""
import numpy as np
import pytest

import sph_b200 as S

pytestmark = pytest.mark.gpu


def _check(oracle, case, pos, typ):
    cfg = case.cfg
    pad = max(0.05, 1.1 * cfg.kernel_scale * cfg.h)      # the grid holds every image
    cfg.grid_lo[:] = [-pad, -pad]
    cfg.grid_hi[:] = [1.0 + pad, 1.0 + pad]
    ext = oracle.periodic_images(cfg, pos, case.vel, case.rho, case.mass, typ, cap=10 * case.n + 64)
    ref = oracle.find_particle_pair(cfg, ext[0], ext[4], pair_cap=400 * case.n)
    key = np.lexsort((ref["pair_j"], ref["pair_i"]))
    with S.Simulation(cfg, case.n) as sim:
        sim.set_state(pos, case.vel, case.rho, case.mass, typ)
        for _ in range(2):                       # the second call reuses the set-up buffers
            got = sim.find_particle_pair(ref["pair_number"] + 64)
            assert got["pair_number"] == ref["pair_number"]
            assert np.array_equal(got["pair_i"], ref["pair_i"][key])
            assert np.array_equal(got["pair_j"], ref["pair_j"][key])


@pytest.mark.parametrize("side", [4, 5, 6, 9, 31, 32, 33, 45, 46, 65])
def test_pairs_at_block_edges_and_thin_boxes(lib, oracle, side):
    case = S.make_tgv(side, jitter=0.1, seed=side)
    _check(oracle, case, case.pos, case.type)


def test_pairs_with_unbinned_particles(lib, oracle):
    case = S.make_tgv(40, jitter=0.1, seed=3)
    typ = case.type.copy()
    typ[::7] = S.TYPE_ILL
    _check(oracle, case, case.pos, typ)


def test_pairs_in_crowded_and_empty_cells(lib, oracle):
    """A quarter of the box squeezed to 2/3 of its width: about 60 neighbours there, gaps beside it."""
    case = S.make_tgv(48, jitter=0.1, seed=4)
    pos = case.pos.copy()
    n = case.n
    pos[:n] = np.where(pos[:n] < 0.25, pos[:n] * (2.0 / 3.0), pos[:n])
    _check(oracle, case, pos, case.type)


def test_images_follow_a_particle_through_the_boundary(lib, oracle):
    """Positions outside the box are wrapped before the images are made."""
    case = S.make_tgv(24, jitter=0.1, seed=5)
    n = case.n
    pos = case.pos + 0.013
    wrapped = np.where(pos > 1.0, pos - 1.0, pos)
    case.cfg.grid_lo[:] = [-0.2, -0.2]
    case.cfg.grid_hi[:] = [1.2, 1.2]
    out = []
    for p in (pos, wrapped):
        with S.Simulation(case.cfg, n) as sim:
            sim.set_state(p, case.vel, case.rho, case.mass, case.type)
            out.append(sim.find_particle_pair(20 * n))
    assert np.array_equal(out[0]["pair_i"], out[1]["pair_i"]) and np.array_equal(out[0]["pair_j"], out[1]["pair_j"])


@pytest.mark.parametrize("side", [40, 260])
def test_pairs_of_typed_particles_under_the_same_boundary_rule(lib, oracle, side):
    """Every type the rule tells apart, on both list builders (8 lanes per particle at
    40^2, a thread at 260^2): only the boundary types look at their candidates' types."""
    case = S.make_tgv(side, jitter=0.1, seed=7)
    case.cfg.pair_rule = S.PAIRS_NO_SAME_BND
    typ = np.random.default_rng(side).choice(np.array([2, -2, -3, -201, -102], case.type.dtype), case.n)
    _check(oracle, case, case.pos, typ)
