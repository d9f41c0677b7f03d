"""The layout kernels (solver.cu): values whose pair parts are zero, subnormal,
huge or infinite come back exactly (a field of equal values is its own fixed point),
the replace-update's caps hold on rows that end inside a block of 32, and a context
that takes over another's memory does not see what that left there."""
import numpy as np
import pytest

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api
from pdfs_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (31, 3, 2), (32, 9, 8), (33, 8, 17), (127, 2, 9), (129, 7, 5)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("v", [0.0, 1e-44, 1e-39, 0.1, 1.0 + 2.0**-30, 3e38, np.inf])
def test_pair_field_of_equal_values_is_stored_exactly(shape, v):
    nx, ny, nz = shape
    f = np.full((nz + 2, ny + 2, nx + 2), v)
    out = np.zeros_like(f)
    with api.Context(nx, ny, nz, (1.0, 1.0, 1.0), precision=L.PREC_FP64, arith=L.ARITH_PAIR) as c:
        c.load(f)
        c.sweep(1)
        c.store(out)
    hi = np.float32(v)
    exp = float(hi) + (float(np.float32(v - float(hi))) if np.isfinite(v) else 0.0)
    exp = np.full_like(f, exp)
    exp[[0, -1]] = exp[:, [0, -1]] = exp[:, :, [0, -1]] = v  # the halo: the input
    assert out.tobytes() == exp.tobytes()


@pytest.mark.parametrize("shape", SHAPES[1:])
def test_polish_caps_and_recycled_memory(shape):
    """The replace-update never exceeds the input (its caps, by block minima), and a
    context on the memory of one that held NaN gives the same bits as a fresh one."""
    w = W.random_spheres(*shape, 1.0, 1.0, 1.0, 2, 1.0, 4.0, seed=sum(shape))
    w.field[1, 1, 1] = 0.25
    r = np.random.default_rng(3)
    f = np.minimum(w.field, r.uniform(0.5, 6.0, w.field.shape))
    kw = dict(frozen=w.frozen, freeze=L.FREEZE_MASK, precision=L.PREC_FP32_POLISH64, arith=L.ARITH_PAIR, tol=1e-5)
    outs = []
    for k in range(2):
        a = f.copy()
        api.solve(a, (1.0, 1.0, 1.0), **kw)
        outs.append(a.tobytes())
        if k == 0:
            nan = np.full_like(f, np.nan)
            api.solve(nan, (1.0, 1.0, 1.0), precision=L.PREC_FP64, fixed_sweeps=1, arith=L.ARITH_PAIR)
    assert outs[0] == outs[1]
    assert (a <= f * (1 + 2.0**-23)).all()
