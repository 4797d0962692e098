"""Resident CG solves of two contexts on two host threads at a time: grids whose plans share a kernel but not its shared
memory (64^3 asks for 49,664 bytes of the four-cell FP64 form, 64 x 48 x 33 for 20,832) must not get in each other's
way, and each solve gives the bits that it gives alone.  In a child process whose cudaLaunchCooperativeKernel waits a
moment before it goes on, so that the other thread's preparation falls between."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SLOW = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
#include <unistd.h>
typedef struct { unsigned x, y, z; } Dim;
typedef int (*Launch)(const void*, Dim, Dim, void**, size_t, void*);
int cudaLaunchCooperativeKernel(const void* f, Dim g, Dim b, void** args, size_t smem, void* stream) {
  Launch next = (Launch)dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaLaunchCooperativeKernel");
  usleep(300);
  return next(f, g, b, args, smem, stream);
}
"""

CHILD = r"""
import threading
import numpy as np
import xflow_gb300 as xf
from xflow_gb300 import capi
from xflow_gb300 import workloads as wl

start = threading.Barrier(2)
failures = []

def run(shape):
    ctx = xf.Context(0)
    codes, _ = wl.neumann_box(*[n + 2 for n in shape])
    g = xf.Grid(ctx, codes, *[np.full(n + 1, 1.0 / n) for n in shape])
    A = xf.Operator(g)
    act = codes == 1
    b = np.where(act, np.random.default_rng(7).standard_normal(codes.shape), 0.0)
    b[act] -= b[act].mean()
    bv, x = g.vec(b), g.vec(None)
    first = None
    start.wait()
    for _ in range(300):
        x.fill(0.0)
        try:
            st = xf.solve(A, x, bv, method=xf.XF_CG, rtol=1e-9, maxit=2)
        except xf.XFError as e:
            failures.append((shape, str(e)))
            break
        if (st.status, st.reserved[0]) != (capi.XF_MAXIT, 2.0):
            failures.append((shape, st.status, st.reserved[0]))
        if first is None:
            first = x.download()
    if first is not None and not np.array_equal(first, x.download()):
        failures.append((shape, "other bits"))

threads = [threading.Thread(target=run, args=(s,)) for s in ((64, 64, 64), (64, 48, 33))]
for t in threads:
    t.start()
for t in threads:
    t.join()
assert not failures, failures
print("OK")
"""


def test_two_contexts_on_two_threads(tmp_path):
    src, lib = os.path.join(tmp_path, "slow.c"), os.path.join(tmp_path, "libslow.so")
    with open(src, "w") as f:
        f.write(SLOW)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", lib, src, "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=lib, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("OK"), r.stdout + r.stderr[-3000:]
