"""Solves around a cudaDeviceReset, on the GPU (in a child process: a reset ends its other
CUDA state): the pools' streams and memory from before it are not used after it, and the
results are the same."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import ctypes as C, sys
sys.path.insert(0, %r)
from pdfs_gb300 import _lib as L, api, workloads as W
def solves():
    out = []
    for n in (30, 44):
        w = W.random_spheres(n, n, n, 1.0, 1.0, 1.0, 3, 2.0, 8.0, seed=2)
        for kw in (dict(precision=L.PREC_FP64, tol=1e-9), dict(precision=L.PREC_FP32_POLISH64, arith=L.ARITH_PAIR,
                                                               scheduler=L.SCHED_OCTANT, tol=1e-5)):
            a = w.field.copy()
            api.solve(a, (1.0, 1.0, 1.0), frozen=w.frozen, freeze=L.FREEZE_MASK, **kw)
            out.append(a.tobytes())
    b = [w.field.copy() for _ in range(3)]
    api.solve_batch(b, [(1.0, 1.0, 1.0)] * 3, frozen=[w.frozen] * 3, freeze=L.FREEZE_MASK, precision=L.PREC_FP32)
    return out + [x.tobytes() for x in b]
first = solves()
assert C.CDLL("libcudart.so.13").cudaDeviceReset() == 0
assert solves() == first
print("ok")
"""


def test_solves_around_a_reset():
    r = subprocess.run([sys.executable, "-c", CODE % ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["ok"], r.stdout + r.stderr[-2000:]
