"""The workspace of the tridiagonal lines: sweeps over the three axes of a box allocate once, in either order, and none
needs more than a box of coefficients.  In a child process whose cudaMalloc counts and can refuse; every result bit for
bit the oracle's."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MALLOC = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int calls;
size_t limit = (size_t)-1;   /* cudaErrorMemoryAllocation above it */
typedef int (*Malloc)(void**, size_t);
int cudaMalloc(void** p, size_t n) {
  Malloc next = (Malloc)dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaMalloc");
  calls++;
  return n > limit ? 2 : next(p, n);
}
"""

CHILD = r"""
import ctypes, sys
import numpy as np
import xflow_gb300 as xf
from oracle import oracle as O
from xflow_gb300 import workloads as wl
lib = ctypes.CDLL(sys.argv[1])
calls, limit = ctypes.c_int.in_dll(lib, "calls"), ctypes.c_size_t.in_dll(lib, "limit")
shape = (20, 20, 20)

def sweep(ctx, axis, seed, most=2**64 - 1):
    codes, nrm = wl.neumann_box(*shape)
    g = xf.Grid(ctx, codes, *(np.full(n - 1, 1.0) for n in shape), nrm)
    rng = np.random.default_rng(seed)
    a, c = rng.uniform(-1, 0, shape), rng.uniform(-1, 0, shape)
    b, f, u = 2.5 + rng.uniform(0, 1, shape), rng.standard_normal(shape), rng.standard_normal(shape)
    v = [g.vec(t) for t in (u, a, b, c, f)]
    M, *where = xf.box_lines(shape, axis)
    before, limit.value = calls.value, most
    xf.thomas_lines(ctx, M, *v, *where)
    ctx.synchronize()
    limit.value = 2**64 - 1
    made = calls.value - before
    W, A, B, C, F = (np.moveaxis(t, axis - 1, -1) for t in (u, a, b, c, f))
    for at in np.ndindex(W.shape[:-1]):
        W[at] = O.thomas(M, W[at], A[at], B[at], C[at], F[at])
    np.testing.assert_array_equal(v[0].download(), u)
    return made

for order in ((1, 2, 3), (2, 3, 1), (3, 1, 2)):
    ctx = xf.Context(0)
    assert [sweep(ctx, axis, axis) for axis in order] == [1, 0, 0]
    ctx.close()
ctx = xf.Context(0)
for axis in (3, 1, 3, 2):
    sweep(ctx, axis, axis, most=110000)   # a box of 19 x 400 doubles, not two
sweep(ctx, 3, 5)
ctx.close()
print("OK")
"""


def test_workspace(tmp_path):
    src, lib = os.path.join(tmp_path, "m.c"), os.path.join(tmp_path, "libm_.so")
    with open(src, "w") as f:
        f.write(MALLOC)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", lib, src, "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=lib, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD, lib], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("OK"), r.stdout + r.stderr[-3000:]
