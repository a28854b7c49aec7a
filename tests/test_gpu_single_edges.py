"""The one-component step kernel at the sizes where its layout can go wrong:
remainders of the 32-wide and 16- or 8-row tiles, boxes narrower than the ring,
the smallest ones, pieces that end inside a column, with and without solid
nodes.  FP64 against the CPU oracle, the same sums in another order: 1e-10
rel-L2; FP32 within the 1e-5 that the FP32 path is held to."""
import numpy as np
import pytest

from cases import _random_moments, rel_l2
from lbfast_b200.capi import Params, Solver
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,highorder,smag", [(15, 0, 0), (19, 0, 1), (27, 0, 0), (27, 1, 1)])
@pytest.mark.parametrize("box,tile,zseg", [
    ((1, 1, 1), 0, 0), ((32, 16, 8), 8, 3), ((33, 17, 9), 16, 0), ((31, 15, 5), 16, 2), ((65, 8, 13), 8, 0),
    ((2, 33, 4), 0, -2), ((96, 49, 7), 0, 0)])
@pytest.mark.parametrize("storage,solid", [("f64", False), ("f64", True), ("f32", False), ("f32", True)])
def test_one_component(lattice, highorder, smag, box, tile, zseg, storage, solid):
    if storage == "f64" and tile == 16:
        tile = 8
    lx, ly, lz = box
    walls = solid and ly > 4
    p = Params(lx=lx, ly=ly, lz=lz, pbc_y=0 if walls else 1, lattice=lattice, highorder=highorder, smagorinsky=smag,
               obstacles=int(solid), visc1=0.05, fx=1e-5, fy=-4e-6, storage=storage, tile_y=tile, zseg=zseg)
    rng = np.random.default_rng(lx * 1000 + ly * 10 + lz)
    block = np.zeros(p.shape, dtype=bool)
    if solid and min(box) > 4:
        block[1:3, 2:4, 1:4] = True
    isf = O.mark_isfluid(block, (1, p.pbc_y, 1), lattice, bool(solid))
    m = np.where((isf == 0)[None], 0.0, _random_moments(rng, p.shape))
    s = Solver(p)
    if solid:
        s.set_isfluid(isf)
    s.set_fields(m)
    s.step(5)
    mg, _, ug = s.get_fields()
    s.close()
    o = O.Oracle(p.oracle_dict(), "f64")
    o.set_isfluid(isf)
    o.set_fields(m, None)
    o.step(5)
    mo, _, _ = o.get_fields()
    fluid = np.abs(isf) == 1
    assert rel_l2(mg, mo, fluid) < (1e-10 if storage == "f64" else 1e-5)


@pytest.mark.parametrize("lattice,highorder", [(15, 0), (19, 0), (27, 1)])
@pytest.mark.parametrize("box,tile,zseg", [((33, 17, 9), 16, 0), ((31, 15, 5), 8, 2), ((65, 8, 13), 16, -4)])
@pytest.mark.parametrize("storage,half_ulp", [("f16", 2.0 ** -12), ("bf16", 2.0 ** -9)])
def test_one_component_16_bit(lattice, highorder, box, tile, zseg, storage, half_ulp):
    """With walls and a solid block.  Every step rounds the six stored Pi - u u
    by at most half an ulp; what it changes relaxes in the steps after it: at
    most `steps` half ulps of the result (P and u are kept in 32 bits)."""
    lx, ly, lz = box
    steps = 5
    p = Params(lx=lx, ly=ly, lz=lz, pbc_y=0, lattice=lattice, highorder=highorder, obstacles=1, visc1=0.05, fx=1e-5,
               storage=storage, tile_y=tile, zseg=zseg)
    rng = np.random.default_rng(lx * 1000 + ly * 10 + lz)
    block = np.zeros(p.shape, dtype=bool)
    block[1:3, 2:4, 1:4] = True
    isf = O.mark_isfluid(block, (1, 0, 1), lattice, True)
    m = np.where((isf == 0)[None], 0.0, _random_moments(rng, p.shape))
    s = Solver(p)
    s.set_isfluid(isf)
    s.set_fields(m)
    s.step(steps)
    mg, _, _ = s.get_fields()
    s.close()
    o = O.Oracle(p.oracle_dict(), "f64")
    o.set_isfluid(isf)
    o.set_fields(m, None)
    o.step(steps)
    mo, _, _ = o.get_fields()
    assert rel_l2(mg, mo, np.abs(isf) == 1) < steps * half_ulp
