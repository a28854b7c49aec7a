"""Random states of every kernel class of the step, and the CRC-32 of their
fields after two steps: shared by test_gpu_step_bits.py and the script that
makes its golden file."""
import zlib

import numpy as np

import lbfast_b200 as L

SHAPE = (9, 30, 40)


def classes():
    """(storage, lattice, highorder, components, smagorinsky, tile rows, served): components 0 one, 1 two, 2 two with DENSRATIO."""
    out = []
    for st in ("f32", "f16", "bf16", "f64"):
        for lat, ho in ((15, 0), (19, 0), (27, 0), (27, 1)):
            for tc in (0, 1, 2):
                for smag in (0, 1):
                    for tile in (8, 16):
                        if st == "f64" and tile == 16:
                            continue
                        # with two components and HIGHORDER in 8-row tiles, which a run takes only
                        # by name, the compiler contracts the collision in another way from build
                        # to build: held to the 16-row tiles within 1e-6 (FP32) and 1e-3 (16-bit)
                        # of the result by test_gpu_parity.py's test of the tile heights
                        if ho and tc and tile == 8 and st != "f64":
                            continue
                        out.append((st, lat, ho, tc, smag, tile, False))
        out.append((st, 27, 1, 2, 0, 8, True))
    return out


def name(c):
    return "%s D3Q%d%s %s%s t%d%s" % (c[0], c[1], "HO" if c[2] else "", ("1c", "2c", "2c_dr")[c[3]], " smag" if c[4] else "",
                                      c[5], " served" if c[6] else "")


def crc(c):
    st, lat, ho, tc, smag, tile, served = c
    rng = np.random.default_rng(5)
    dt = np.float64 if st == "f64" else np.float32
    m = np.empty((10,) + SHAPE, dt)
    m[0] = rng.uniform(-.01, .01, SHAPE)
    m[1:4] = rng.uniform(-.05, .05, (3,) + SHAPE)
    u, v, w = m[1:4]
    m[4:] = np.array([u * u, v * v, w * w, u * v, u * w, v * w]) + rng.uniform(-1e-3, 1e-3, (6,) + SHAPE).astype(dt)
    phi = rng.uniform(0, 1, SHAPE).astype(dt) if tc else None
    kw = dict(twocomponent=1, densratio=int(tc == 2), visc2=0.03, rho_r=2.0, rho_b=1.0, sigma=0.01, width=4.0,
              tau_diff=0.1) if tc else {}
    p = L.Params(lx=SHAPE[2], ly=SHAPE[1], lz=SHAPE[0], lattice=lat, highorder=ho, storage=st, visc1=0.01, smagorinsky=smag,
                 fx=1.3e-4, fy=-2.1e-4, fz=3.7e-4, tile_y=tile, **kw)
    if served:
        with L.Server(chunk=2) as s:
            i = s.submit(p, m, phi, 2)
            s.drain()
            fields = s.fetch(i)
    else:
        s = L.Solver(p)
        s.set_fields(m, phi)
        s.step(2)
        fields = s.get_fields(dtype=dt)
        s.close()
    crc = 0
    for f in fields:
        if f is not None:
            crc = zlib.crc32((np.ascontiguousarray(f) + dt(0)).tobytes(), crc)  # -0 as 0
    return crc
