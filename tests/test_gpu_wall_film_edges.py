"""Sizes at which the film-repulsion search and the wall passes can go wrong:
edges of the search's 16 x 8 x 8 tiles, boxes smaller than its window, open
axes of three nodes.  FP64 against the CPU oracle, the same sums in another
order: 1e-10 rel-L2."""
import numpy as np
import pytest

from cases import _blobs, _random_moments, rel_l2
from lbfast_b200.capi import Params, Solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _compare(p, isf, m, phi, nsteps):
    s = Solver(p)
    if p.obstacles:
        s.set_isfluid(isf)
    s.set_fields(m, phi)
    s.step(nsteps)
    mg, pg, _ = s.get_fields()
    s.close()
    o = O.Oracle(p.oracle_dict(), "f64")
    o.set_isfluid(isf)
    o.set_fields(m, phi)
    o.step(nsteps)
    mo, po, _ = o.get_fields()
    fluid = np.abs(isf) == 1
    assert rel_l2(mg, mo, fluid) < 1e-10
    if p.twocomponent:
        assert rel_l2(pg, po, fluid) < 1e-10


@pytest.mark.parametrize("box,pbc,q_th,cos", [
    ((16, 8, 8), (1, 1, 1), 0.05, -0.5), ((17, 9, 7), (1, 1, 1), 0.05, -0.5), ((33, 15, 18), (1, 0, 1), 0.02, -0.2),
    ((5, 4, 3), (1, 1, 1), 0.01, 0.3), ((40, 24, 16), (0, 1, 1), 0.15, -0.9), ((18, 10, 12), (1, 1, 0), 0.0, 0.5)])
def test_film_search(box, pbc, q_th, cos):
    lx, ly, lz = box
    rng = np.random.default_rng(lx * 100 + ly)
    p = Params(lx=lx, ly=ly, lz=lz, pbc_x=pbc[0], pbc_y=pbc[1], pbc_z=pbc[2], lattice=27, twocomponent=1, densratio=1,
               visc1=0.05, visc2=0.08, rho_r=1.0, rho_b=0.5, sigma=0.01, width=2.5, tau_diff=0.1, storage="f64",
               repulsive_flux=1, a_rep=0.05, cos_opp_t=cos, q_th=q_th)
    phi = _blobs(rng, p.shape, 6, 2.0, 4.0, 2.5)
    m = _random_moments(rng, p.shape, amp_u=0.002, amp_p=0.0005, amp_neq=1e-6)
    _compare(p, np.ones(p.shape, np.int8), m, phi, 3)


@pytest.mark.parametrize("box,pbc,bb,types", [
    ((3, 12, 9), (0, 1, 1), 0, ((1, 1), (0, 0), (0, 0))), ((3, 3, 14), (0, 0, 1), 1, ((0, 0), (1, 2), (0, 0))),
    ((20, 11, 3), (1, 1, 0), 1, ((0, 0), (0, 0), (0, 0))), ((33, 9, 8), (0, 0, 0), 1, ((1, 2), (0, 0), (0, 0)))])
@pytest.mark.parametrize("lattice,highorder", [(15, 0), (19, 0), (27, 1)])
def test_wall_passes(box, pbc, bb, types, lattice, highorder):
    lx, ly, lz = box
    rng = np.random.default_rng(lx * 100 + lz)
    p = Params(lx=lx, ly=ly, lz=lz, pbc_x=pbc[0], pbc_y=pbc[1], pbc_z=pbc[2], lattice=lattice, highorder=highorder,
               obstacles=1, bounce_back=bb, visc1=0.1, storage="f64", openbc=1, openbc_type=types,
               openbc_press=((0.002, -0.002),) * 3, fx=1e-6)
    solid = np.zeros(p.shape, dtype=bool)
    if min(box) > 3:
        solid[3:5, 3:6, 10:14] = True
    isf = O.mark_isfluid(solid, pbc, lattice, True)
    m = np.where((isf == 0)[None], 0.0, _random_moments(rng, p.shape, amp_u=0.003, amp_p=0.002))
    _compare(p, isf, m, None, 4)


@pytest.mark.parametrize("box,pbc,corr", [((17, 16, 9), (1, 0, 1), 0), ((33, 10, 15), (1, 0, 1), 1), ((16, 17, 8), (0, 1, 1), 1),
                                          ((31, 9, 17), (1, 1, 1), 1)])
def test_film_search_around_solid_nodes(box, pbc, corr):
    """Solid nodes across the edges of the search's tiles, with and without the mass correction."""
    lx, ly, lz = box
    rng = np.random.default_rng(lx * 100 + ly)
    p = Params(lx=lx, ly=ly, lz=lz, pbc_x=pbc[0], pbc_y=pbc[1], pbc_z=pbc[2], lattice=27, twocomponent=1, densratio=1,
               visc1=0.05, visc2=0.08, rho_r=1.0, rho_b=0.5, sigma=0.01, width=2.5, tau_diff=0.1, storage="f64",
               repulsive_flux=1, a_rep=0.05, cos_opp_t=-0.2, q_th=0.02, obstacles=1, phi_correction=corr)
    solid = np.zeros(p.shape, dtype=bool)
    solid[6:9, 6:9, 14:18] = True
    isf = O.mark_isfluid(solid, pbc, 27, True)
    phi = np.where(isf == 0, 0.0, _blobs(rng, p.shape, 6, 2.0, 4.0, 2.5))
    m = np.where((isf == 0)[None], 0.0, _random_moments(rng, p.shape, amp_u=0.002, amp_p=0.0005, amp_neq=1e-6))
    _compare(p, isf, m, phi, 4)


@pytest.mark.parametrize("two,bb", [(0, 0), (0, 1), (1, 0)])
def test_second_set_isfluid(two, bb):
    """The wall links and wetting tables are those of the last isfluid, with more or fewer wall nodes than before."""
    extra = dict(twocomponent=1, densratio=1, visc2=0.08, rho_r=1.0, rho_b=0.5, sigma=0.01, width=2.5, tau_diff=0.1) if two else {}
    p = Params(lx=34, ly=12, lz=10, pbc_y=0, lattice=19, obstacles=1, bounce_back=bb, visc1=0.05, fx=1e-5, storage="f32", **extra)
    rng = np.random.default_rng(4)
    m, phi = _random_moments(rng, p.shape), _blobs(rng, p.shape, 3, 2.0, 3.0, 2.5)
    solid = np.zeros(p.shape, dtype=bool)
    few = O.mark_isfluid(solid, (1, 0, 1), 19, True)
    solid[3:7, 4:8, 5:30] = True
    many = O.mark_isfluid(solid, (1, 0, 1), 19, True)

    def run(geometries):
        s = Solver(p)
        for isf in geometries:
            s.set_isfluid(isf)
            s.set_fields(np.where((isf == 0)[None], 0.0, m), phi if two else None)
            s.step(3)
        out = s.get_fields()
        s.close()
        return out

    for a, b in ((few, many), (many, few)):
        for x, y in zip(run([a, b]), run([b])):
            assert (x is None and y is None) or np.array_equal(x, y, equal_nan=True)
