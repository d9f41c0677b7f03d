"""Plain sweeps of grids of many bricks, whose tickets follow the node levels, and mixed
sweeps of grids thin in y, which run on pencils: the bits of the selectable brick tiles,
whose tickets follow the brick levels, after orderings from opposite corners."""
import numpy as np
import pytest

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api

pytestmark = pytest.mark.gpu

CASES = [((1500, 4, 1500), dict(precision=L.PREC_FP32), 10, 9),
         ((251, 233, 241), dict(precision=L.PREC_FP32), 10, 9),
         ((1200, 4, 1200), dict(precision=L.PREC_FP64), 6, 5),
         ((5, 1200, 1201), dict(precision=L.PREC_FP64, arith=L.ARITH_FAST), 6, 5),
         ((2000, 4, 2001), dict(precision=L.PREC_FP64, arith=L.ARITH_PAIR), 6, 5),
         ((1000, 250, 257), dict(precision=L.PREC_FP64, arith=L.ARITH_MIXED), 6, 5),
         ((1000, 4, 1000), dict(precision=L.PREC_FP64, arith=L.ARITH_MIXED), 6, 5)]


@pytest.mark.parametrize("shape,kw,tile,ref", CASES)
def test_sweeps_equal_brick_tile(shape, kw, tile, ref):
    nx, ny, nz = shape
    r = np.random.default_rng(sum(shape))
    f = np.full((nz + 2, ny + 2, nx + 2), 1e10)
    n = nx * ny * nz // 5000
    f[r.integers(1, nz + 1, n), r.integers(1, ny + 1, n), r.integers(1, nx + 1, n)] = r.uniform(0, 1, n)
    out = []
    for t in (tile, ref):
        t = t if kw["precision"] == L.PREC_FP32 else t << 8
        a = np.empty_like(f)
        with api.Context(nx, ny, nz, (1.0, 1.0, 1.0), tile=t, **kw) as c:
            c.load(f)
            for sn in (1, 2, 6):
                c.sweep(sn)
            c.store(a)
        out.append(a)
    assert np.array_equal(*out)
