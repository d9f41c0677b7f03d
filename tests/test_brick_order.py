"""The ticket order of plain sweeps' bricks (host code on a fake CUDA runtime, no GPU):
the list that a context copies to the device names every brick once, each after its
three upwind neighbours, and on a grid of many bricks by the node level at which a
brick can start -- so that the bricks taken together are those that run together."""
import numpy as np
import pytest

import fakecuda
from pdfs_gb300 import _lib as L

SHIM = """
import ctypes as C, os
o = dict(%r)
with api.Context(*%r, (1.0, 1.0, 1.0), **o) as c:
    pass
"""


def order(shape, kw, b, bz):
    """The plain sweeps' list: the host-to-device copy of one int a brick."""
    nt = [-(-n // m) for n, m in zip(shape, (b, b, bz))]
    n = nt[0] * nt[1] * nt[2]
    got = fakecuda.copies(SHIM % (list(kw.items()), shape), n * 4)
    assert got
    return nt, np.frombuffer(got[-1], np.int32)


CASES = [((2000, 4, 2000), dict(precision=L.PREC_FP32), 8, 32, 4),
         ((2000, 4, 2000), dict(precision=L.PREC_FP64), 8, 16, 2),
         ((2000, 4, 2000), dict(precision=L.PREC_FP64, arith=L.ARITH_PAIR), 16, 32, 2),
         ((251, 233, 241), dict(precision=L.PREC_FP32), 8, 32, 4),
         ((2000, 8, 1500), dict(precision=L.PREC_FP64, arith=L.ARITH_PAIR), 16, 32, 2),
         ((500, 8, 500), dict(precision=L.PREC_FP64, arith=L.ARITH_PAIR), 16, 32, 1),
         ((151, 127, 110), dict(precision=L.PREC_FP64), 8, 16, 1),
         ((500, 4, 500), dict(precision=L.PREC_FP64, arith=L.ARITH_FAST), 8, 16, 1)]


@pytest.mark.parametrize("shape,kw,b,bz,wz", CASES)
def test_order(shape, kw, b, bz, wz):
    nt, o = order(shape, kw, b, bz)
    n = nt[0] * nt[1] * nt[2]
    assert sorted(o) == list(range(n))
    i, j, k = o % nt[0], o // nt[0] % nt[1], o // (nt[0] * nt[1])
    assert (np.diff(i + j + wz * k) >= 0).all()  # by start level
    at = np.empty(n, int)
    at[o] = np.arange(n)
    for d, m in ((1, i), (nt[0], j), (nt[0] * nt[1], k)):
        up = m > 0
        assert (at[o[up] - d] < np.arange(n)[up]).all()


@pytest.mark.parametrize("shape,pencils", [((1000, 4, 1000), True), ((2000, 12, 2000), True), ((1000, 24, 1000), True),
                                           ((200, 8, 1000), True), ((1000, 1, 1000), False), ((300, 16, 300), False),
                                           ((1400, 24, 1400), False), ((4, 1000, 1000), False), ((64, 64, 64), False)])
def test_mixed_sweeps_of_thin_grids(shape, pencils):
    code = """
with api.Context(*%r, (1.0, 1.0, 1.0), precision=L.PREC_FP64, arith=L.ARITH_%s, max_sweeps=8) as c:
    c.load(np.zeros(tuple(n + 2 for n in %r)))
    c.run()
"""
    for arith, want in (("MIXED", pencils), ("PAIR", False)):
        _, log = fakecuda.run(code % (shape, arith, shape[::-1]))
        names = [w[1] for w in log if w[0] == "launch"]
        assert any("pc_sweep_kernel" in n for n in names) == want
        assert any("t3_sweep_kernel" in n for n in names) == (not want)
