"""When a state page-locks its buffer for results: once it has been asked often enough that the locking pays, and never for
a served run (the call may wait for all streams of the device).  Counted by a shared object that stands before the runtime's functions, in a child process."""
import os
import subprocess
import sys
import textwrap

import pytest

from tests import decks

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

COUNTER = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int locked, freed;
static void* real(const char* name) { return dlsym(dlopen("libcudart.so.13", RTLD_NOW), name); }
int cudaMallocHost(void** p, size_t n) {
  locked++;
  return ((int (*)(void**, size_t))real("cudaMallocHost"))(p, n);
}
int cudaFreeHost(void* p) {
  freed++;
  return ((int (*)(void*))real("cudaFreeHost"))(p);
}
"""

CHILD = """
import ctypes, sys
sys.path.insert(0, %r)
from epic2d_mcc_gb300 import api as E, workloads
so = ctypes.CDLL(%r)
def count():
    return tuple(ctypes.c_int.in_dll(so, k).value for k in ("locked", "freed"))
sim = E.Simulation.from_ini(%r)
for asked, locked in ((16, 0), (1, 1), (40, 1)):
    for _ in range(asked):
        sim.num_particles(0)
    assert count() == (locked, 0), (asked, count())
sim.close()
assert count() == (1, 1), count()
srv = E.Server(budget_bytes=4 << 30, max_inflight=2, chunk_steps=7)
e, ela, exc, ion = workloads.synthetic_table()
srv.set_log_cross_sections(ela, exc, ion, e[0], e[-1])
ids = [srv.submit(E.make_request(i, steps=9, collisions=c, seed=5, precision=1)) for i, c in %r]
srv.start()
srv.wait(300)
for i in ids:
    assert srv.result(i).status == 0
srv.close()
assert count() == (1, 1), count()
print("counted")
"""


def test_who_page_locks(gpu_lib, tmp_path):
    d = str(tmp_path)
    (tmp_path / "count.c").write_text(COUNTER)
    so = str(tmp_path / "count.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", so, str(tmp_path / "count.c"), "-ldl"], check=True)
    plain = decks.write(decks.deck(ne=500, ni=500, solver="cg"), d)
    three = decks.write(decks.deck(nx=32, ny=32, ne=5000, ni=5000, solver="cg", tol="1e-8", collisions=True,
                                   beam=dict(n=500, t=1, frac=0.1, vx=1, vy=0)), d)
    grids = [dict(type="reactconduct", min_x=10, max_x=12, min_y=4, max_y=16, grid_voltage=10)] + [
        dict(type="circular", x_center=x, y_center=30, electrode_number=4, grid_radius=3, electrod_radius=1,
             electrode_voltage=-5) for x in (20, 30, 40)]
    em = [dict(x0=2, y0=20 + k, x1=2, y1=30, temp=0.5, numparticle=40, vdx=0.2, vdy=0, species_idx1=0, species_idx2=1)
          for k in range(4)]
    walls = decks.write(decks.deck(nx=64, ny=48, ne=5000, ni=5000, bc="open", solver="gs", tol="1e-6", grids=grids,
                                   emitters=em), d)
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(CHILD % (ROOT, so, plain, [(three, True), (walls, False)]))],
                       capture_output=True, text=True, timeout=600, env=dict(os.environ, LD_PRELOAD=so))
    assert r.returncode == 0 and "counted" in r.stdout, r.stdout + r.stderr
