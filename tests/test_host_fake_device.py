"""Host paths around the device, run in a child process against a CUDA runtime
that keeps device memory on the host and launches nothing (fake_cudart.c):
allocations that fail, the memory that an admission holds, the keys of the
schedule cache.  No GPU."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

PRELUDE = """
import ctypes, sys
sys.path[:0] = [{root!r}, {here!r}]
import numpy as np
import lbfast_b200 as L
from lbfast_b200.capi import LBF_OK
fake = ctypes.CDLL({so!r})
fake.fake_launches.restype = fake.fake_peak.restype = ctypes.c_longlong
E_STATE = {state}
def code(f, *a, **k):
    try:
        f(*a, **k)
    except L.LbfError as e:
        return e.code
    return LBF_OK
def isfluid(p):
    f = np.ones(p.shape, np.int8)
    f[:, 0] = f[:, -1] = 0
    f[:, 1] = f[:, -2] = -1
    return f
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-Wall", "-Werror", "-Wno-builtin-declaration-mismatch", "-o", so,
                    os.path.join(HERE, "fake_cudart.c")], check=True)

    def run(body):
        pre = PRELUDE.format(root=os.path.dirname(HERE), here=HERE, so=so, state=-4)
        r = subprocess.run([sys.executable, "-c", pre + body], env=dict(os.environ, LD_PRELOAD=so), capture_output=True,
                           text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


@pytest.mark.parametrize("extra", ["", ", bounce_back=1", ", twocomponent=1, visc2=0.1, width=4.0"])
def test_failed_set_isfluid_leaves_no_half_made_geometry(fake, extra):
    """Whichever of its allocations fails, the handle takes no fields before and
    no step after, and launches nothing; a call that succeeds sets it right."""
    fake("""
p = L.Params(lx=40, ly=12, lz=9, lattice=19, obstacles=1, pbc_y=0, visc1=0.1, storage="f32", tile_y=16%s)
f = isfluid(p)
m, phi = np.zeros((10,) + p.shape, np.float32), np.zeros(p.shape, np.float32) if p.twocomponent else None
failed = 0
for n in range(40):
    s = L.Solver(p)
    fake.fake_fail_alloc(n)
    rc = code(s.set_isfluid, f)
    fake.fake_fail_alloc(-1)
    if rc == LBF_OK:
        s.close()
        break
    failed += 1
    assert code(s.set_fields, m, phi) == E_STATE
    assert code(s.set_isfluid, f) == LBF_OK and code(s.set_fields, m, phi) == LBF_OK and code(s.step, 2) == LBF_OK
    # once more, with tables in place
    fake.fake_fail_alloc(n)
    assert code(s.set_isfluid, f) != LBF_OK
    fake.fake_fail_alloc(-1)
    before = fake.fake_launches()
    assert code(s.step, 2) == E_STATE and fake.fake_launches() == before
    assert code(s.set_isfluid, f) == LBF_OK and code(s.step, 2) == LBF_OK and fake.fake_launches() > before
    s.close()
assert failed >= 2, failed
""" % extra)


def test_admission_during_a_chunk_holds_one_staging_buffer(fake):
    """Solves that are admitted while a chunk runs: the device holds the budget
    and one staging buffer, however many are admitted at once."""
    fake("""
p = L.Params(lx=32, ly=32, lz=32, lattice=27, highorder=1, twocomponent=1, densratio=1, visc1=0.1, visc2=0.1,
             rho_r=2.0, sigma=0.01, width=4.0, tau_diff=0.1, storage="f16")
m, phi = np.zeros((10,) + p.shape, np.float32), np.zeros(p.shape, np.float32)
b, staging = L.Server.solve_bytes(p), m.nbytes
s = L.Server(mem_budget=5 * b + b // 2, chunk=4, use_graph=False)
fake.fake_reset_peak()
base = fake.fake_peak()
long = s.submit(p, m, phi, 40)
ids = [s.submit(p, m, phi, 4) for _ in range(12)]
s.drain()
assert all(s.poll(i)["state"] == "done" for i in [long] + ids)
held = fake.fake_peak() - base
assert held <= 5 * b + staging + 65536, (held / b, staging / b)
s.close()
""")


def test_schedules_are_tuned_per_kernel_class(fake):
    """A class of its own times its own schedules: none takes over one that was
    measured on another kernel of the same box."""
    fake("""
base = dict(lx=64, ly=48, lz=40, lattice=27, highorder=1, twocomponent=1, visc1=0.1, visc2=0.1, sigma=0.01, width=4.0,
            tau_diff=0.1, storage="f32")
def first_step(**kw):
    p = L.Params(**dict(base, **kw))
    s = L.Solver(p)
    s.set_fields(np.zeros((10,) + p.shape, np.float32), np.zeros(p.shape, np.float32))
    n = fake.fake_launches()
    s.step(1)
    n = fake.fake_launches() - n
    s.close()
    return n
assert first_step() > 10
assert first_step() < 5  # the same class again
film = dict(repulsive_flux=1, a_rep=0.05, cos_opp_t=-0.5, q_th=0.05)
for other in (film, dict(phi_correction=1), dict(smagorinsky=1), dict(film, phi_correction=1)):
    assert first_step(**other) > 10, other
    assert first_step(**other) < 8, other
""")
