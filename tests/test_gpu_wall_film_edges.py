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
