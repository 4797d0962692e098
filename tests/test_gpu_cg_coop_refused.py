"""A cooperative launch that the driver refuses sends the solve to the kernel chain: in a child process whose
cudaLaunchCooperativeKernel is a stand-in that always returns an error code, a grid that the resident CG would take is
solved all the same, to the same tolerance, and so is the next one."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#include <stddef.h>
int refused;
/* cudaErrorCooperativeLaunchTooLarge */
int cudaLaunchCooperativeKernel(const void* f, ...) { refused++; return 720; }
"""

CHILD = r"""
import ctypes, sys
import numpy as np
import xflow_gb300 as xf
from xflow_gb300 import capi
from xflow_gb300 import workloads as wl
refused = ctypes.c_int.in_dll(ctypes.CDLL(sys.argv[1]), "refused")
ctx = xf.Context(0)
for shape in ((20, 18, 22), (33, 31, 35)):
    codes, _ = wl.neumann_box(*[n + 2 for n in shape])
    act = codes == 1
    b = np.where(act, np.random.default_rng(1).standard_normal(codes.shape), 0.0)
    b[act] -= b[act].mean()
    for precision in (xf.XF_PREC_FP64, xf.XF_PREC_MIXED):
        g = xf.Grid(ctx, codes, *[np.full(n + 1, 1.0 / n) for n in shape])
        A = xf.Operator(g)
        for again in range(2):
            x = g.vec(np.zeros(codes.shape))
            st = xf.solve(A, x, g.vec(b), method=xf.XF_CG, precision=precision, rtol=1e-9)
            assert st.status == capi.XF_OK and st.rel_resid <= 1e-9, (shape, precision, st.status, st.rel_resid)
            assert st.reserved[0] > 100, st.reserved[0]   # the chain's launches
assert refused.value == 4, refused.value   # once a grid and precision
print("OK")
"""


def test_refused_launch_goes_to_the_chain(tmp_path):
    src, lib = os.path.join(tmp_path, "fake.c"), os.path.join(tmp_path, "libfake.so")
    with open(src, "w") as f:
        f.write(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", lib, src], check=True)
    env = dict(os.environ, LD_PRELOAD=lib, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD, lib], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("OK"), r.stdout + r.stderr[-3000:]
