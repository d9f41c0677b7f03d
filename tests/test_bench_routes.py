"""bench.py names the kernel that runs: plain_kernel against the launches of the library
(host code on a fake CUDA runtime, no GPU) on both sides of every line of the routing."""
import importlib.util
import os
import re

import pytest

import fakecuda
from pdfs_gb300 import _lib as L

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUN = """
with api.Context(*%r, (1.0, 1.0, 1.0), precision=%d, arith=%d, tile=%d, fixed_sweeps=1) as c:
    c._lib.pdfs_ctx_load(c.h, C.c_void_p(0x500000000000), None)
    print(c.run()["tile"])
"""
AR = ["REF", "FAST", "MIXED", "PAIR"]


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_under_test", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def launched(names):
    """The sweep kernel's name as bench.py writes it."""
    for n in names:
        m = re.search(r"(t3|pc|ws|lc)_sweep_kernelI([fd])((?:L[ib]\d+E)*)E", n)
        if m:
            k, t, a = m.group(1), {"f": "float", "d": "double"}[m.group(2)], [int(x) for x in re.findall(r"\d+", m.group(3))]
            if k == "t3":
                a = a[:3] + [["MIN", "REPLACE"][a[3]], AR[a[4]]]
            elif k == "pc":
                a = [["MIN", "REPLACE"][a[0]], AR[a[1]]]
            return "%s_sweep_kernel<%s, %s>" % (k, t, ", ".join(map(str, a)))


@pytest.mark.parametrize("shape", [(64, 64, 64), (250, 250, 900), (2000, 4, 2000), (300, 16, 300), (1400, 24, 1400),
                                   (406, 406, 408), (400, 400, 400)])
@pytest.mark.parametrize("prec,arith,tile", [(1, 0, 0), (0, 0, 0), (0, 1, 0), (0, 2, 0), (0, 3, 0), (1, 0, 9),
                                             (0, 3, 5 << 8), (1, 0, 11)])
def test_plain_kernel(bench, shape, prec, arith, tile):
    text, log = fakecuda.run("import ctypes as C\n" + RUN % (shape, prec, arith, tile), memory=1 << 40)
    got = launched([w[1] for w in log if w[0] == "launch"])
    kind = "fp32" if prec == L.PREC_FP32 else "fp64"
    assert bench.plain_kernel(kind, int(text), prec, arith, *shape) == got
