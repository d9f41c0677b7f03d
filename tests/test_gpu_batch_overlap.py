"""A batch round's sweeps overlap pencil by pencil (a pencil follows its own and its
four neighbours' previous sweep): every grid equals the same number of fixed sweeps
of a lone solve, bit for bit, whatever the shapes beside it -- long in x, y and z,
one pencil, ragged pencils -- and again on the next call, on recycled memory."""
import numpy as np
import pytest

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api
from pdfs_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(150, 33, 20), (20, 150, 41), (33, 40, 140), (16, 16, 16), (17, 31, 64), (1, 97, 3)]


@pytest.mark.parametrize("kw", [dict(precision=L.PREC_FP32, tol=0.0),
                                dict(precision=L.PREC_FP64, arith=L.ARITH_PAIR, tol=1e-5),
                                dict(precision=L.PREC_FP64, arith=L.ARITH_REFERENCE, tol=1e-9)])
def test_rounds_equal_fixed_sweeps(kw):
    ws = [W.random_spheres(*s, 1.0, 1.0, 1.0, 3, 1.5, 8.0, seed=k) for k, s in enumerate(SHAPES)]
    for w in ws:
        w.field[1, 1, 1] = 0.25
    for _ in range(3):
        fields = [w.field.copy() for w in ws]
        st = api.solve_batch(fields, [(1.0, 1.0, 1.0)] * len(ws), frozen=[w.frozen for w in ws],
                             freeze=L.FREEZE_MASK, **kw)
        for w, f, s in zip(ws, fields, st):
            ref = w.field.copy()
            api.solve(ref, (1.0, 1.0, 1.0), frozen=w.frozen, freeze=L.FREEZE_MASK,
                      fixed_sweeps=s["sweeps_fp32"] + s["sweeps_fp64"], **kw)
            assert np.array_equal(f, ref, equal_nan=True), w.name
