"""Kernels' attributes (shared memory beyond 48 KB, clusters of more than eight blocks) belong to a device and its context,
and a launch may be refused.  A shared object before the runtime's functions keeps count in a child process: it refuses,
on the host, launches whose attributes have not been set since it was told to forget them (as another device would), or
every cluster; and the device is reset.  The answers stay the same: bit for bit, or, where another kernel takes a refused
solve, the same iterates to rounding."""
import os
import subprocess
import sys
import textwrap

import pytest

from tests import decks

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>
static struct { const void* f; int smem, wide; } seen[64];
static int n_seen, pending;
int refuse_clusters, refused;
static void* real(const char* name) { return dlsym(dlopen("libcudart.so.13", RTLD_NOW), name); }
static int at(const void* f) {
  int k = 0;
  while (k < n_seen && seen[k].f != f) k++;
  if (k == n_seen && n_seen < 63) seen[n_seen++].f = f;
  return k;
}
void forget(void) {
  for (int k = 0; k < 64; k++) seen[k].smem = seen[k].wide = 0;
}
int most_smem(void) {
  int m = 0;
  for (int k = 0; k < n_seen; k++) m = seen[k].smem > m ? seen[k].smem : m;
  return m;
}
static cudaError_t no(void) {
  refused++;
  return pending = cudaErrorInvalidClusterSize;
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) seen[at(f)].smem = v;
  if (a == cudaFuncAttributeNonPortableClusterSizeAllowed) seen[at(f)].wide = v;
  return ((cudaError_t (*)(const void*, enum cudaFuncAttribute, int))real("cudaFuncSetAttribute"))(f, a, v);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  unsigned wide = 1;
  for (unsigned k = 0; k < c->numAttrs; k++)
    if (c->attrs[k].id == cudaLaunchAttributeClusterDimension) wide = c->attrs[k].val.clusterDim.x;
  const int k = at(f);
  if ((refuse_clusters && wide > 1) || (wide > 8 && !seen[k].wide) ||
      (c->dynamicSmemBytes > 48 * 1024 && (int)c->dynamicSmemBytes > seen[k].smem))
    return no();
  return ((cudaError_t (*)(const cudaLaunchConfig_t*, const void*, void**))real("cudaLaunchKernelExC"))(c, f, args);
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 g, dim3 b, void** args, size_t smem, cudaStream_t s) {
  if (smem > 48 * 1024 && (int)smem > seen[at(f)].smem) return no();
  return ((cudaError_t (*)(const void*, dim3, dim3, void**, size_t, cudaStream_t))real("cudaLaunchCooperativeKernel"))(
      f, g, b, args, smem, s);
}
cudaError_t cudaGetLastError(void) {
  const int e = pending;
  pending = 0;
  return e ? (cudaError_t)e : ((cudaError_t (*)(void))real("cudaGetLastError"))();
}
"""

CHILD = """
import ctypes, sys
import numpy as np
sys.path.insert(0, %r)
from epic2d_mcc_gb300 import api as E
L = E.lib()
rt = ctypes.CDLL("libcudart.so.13")
shim = ctypes.CDLL(%r)
refuse, refused = (ctypes.c_int.in_dll(shim, k) for k in ("refuse_clusters", "refused"))
vp, i32, f64 = ctypes.c_void_p, ctypes.c_int, ctypes.c_double
L.epic_last_error.restype = ctypes.c_char_p
fn = L.epic_pcg_solve_static
fn.argtypes = [vp, vp, i32, i32, f64, f64, f64, i32, vp, ctypes.POINTER(i32), ctypes.POINTER(f64)]
hold = []

def static(n):
    rho, phi = np.random.default_rng(n).normal(size=n * n), np.empty(n * n)
    size = ctypes.c_size_t(8 * n * n)
    rho_d, phi_d, it, err = vp(), vp(), i32(), f64()
    for p in (rho_d, phi_d):
        assert rt.cudaMalloc(ctypes.byref(p), size) == 0
        hold.append(p)
    assert rt.cudaMemcpy(rho_d, rho.ctypes.data_as(vp), size, 1) == 0
    st = fn(rho_d, phi_d, n, n, 1.0, 1.0, 1e-8, 10000, None, ctypes.byref(it), ctypes.byref(err))
    assert st == 0, (st, L.epic_last_error())
    assert rt.cudaMemcpy(phi.ctypes.data_as(vp), phi_d, size, 2) == 0
    return it.value, phi

def state(ini):
    sim = E.Simulation.from_ini(ini)
    sim.set_grid("rho", np.random.default_rng(1).normal(size=sim.nx * sim.ny))
    it, _, _ = sim.potential_solver()
    phi = sim.grid("phi")
    sim.close()
    return it, phi

def answers():
    return [static(n) for n in (20, 60, 200)] + [state(i) for i in %r]

def same(b, exact):
    for k, (x, y) in enumerate(zip(first, b)):
        assert x[0] == y[0], (k, x[0], y[0])
        if k in exact:
            assert np.array_equal(x[1], y[1]), k
        else:
            assert np.max(np.abs(x[1] - y[1])) <= 1e-12 * np.max(np.abs(x[1])), k

first = answers()
every = range(len(first))
assert refused.value == 0
shim.forget()
same(answers(), every)          # every launch sets what it needs
assert refused.value == 0
for k, ini in enumerate(%r):    # plain launches: seen by the attribute
    sim = E.Simulation.from_ini(ini)
    shim.forget()
    sim.set_grid("rho", np.zeros(sim.nx * sim.ny))
    sim.potential_solver()
    assert shim.most_smem() > 48 * 1024
    sim.close()
refuse.value = 1
same(answers(), %r)
assert refused.value > 0
refuse.value = 0
del hold[:]
assert rt.cudaDeviceReset() == 0
same(answers(), every)
print("same")
"""


def test_attributes_and_refusals(gpu_lib, tmp_path):
    def ini(nx, ny, solver, extra=""):
        return decks.write(decks.deck(nx=nx, ny=ny, ne=1000, ni=1000, solver=solver, tol="1e-6", maxit=60,
                                      solver_extra=extra), str(tmp_path))

    per, wx = "poisson_bc = periodic\n", "poisson_bc = dirichlet_x\n"
    inis = [ini(60, 60, "cg"), ini(2046, 20, "cg"), ini(64, 64, "gs"), ini(64, 64, "gshybrid"), ini(120, 130, "gs", per),
            ini(200, 180, "gs"), ini(200, 180, "gs", per), ini(6, 2000, "gs", wx)]
    (tmp_path / "shim.c").write_text(SHIM)
    so = str(tmp_path / "shim.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-o", so, str(tmp_path / "shim.c"), "-ldl"],
                   check=True)
    sor = [3 + k for k in (2, 4, 5, 6, 7)]
    code = CHILD % (ROOT, so, inis, [inis[4]], sor)
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(code)], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, LD_PRELOAD=so))
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
