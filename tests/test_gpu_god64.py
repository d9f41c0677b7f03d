"""The FP64 solvers with few FP64-pipe operations (god64.cuh: the plain FP64
sweeps on bricks) against the plain solvers of the column kernel.  Reference
arithmetic: the same bits, for ordinary fields, for infinities, NaN, negative and
huge values, and for spacings that push discriminants and quotients out of the
fast paths' ranges.  Fast arithmetic: a node's rounding may differ by some units in
the last place (four roundings moved, each 2^-53, at a sensitivity below 4 at a
node) and a value passes through at most 8 (nx + ny + nz) nodes in 8 orderings."""
import numpy as np
import pytest

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api
from pdfs_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (8, 8, 16), (9, 8, 17), (7, 15, 15), (8, 1, 33), (33, 50, 8), (50, 43, 52)]
SPACINGS = [(1.0, 1.0, 1.0), (0.7, 1.3, 0.4), (1.0 / 63, 1.0 / 63, 1.0 / 31)]


def sweeps(field, frozen, sp, arith, tile):
    nz, ny, nx = (n - 2 for n in field.shape)
    out = np.empty_like(field)
    with api.Context(nx, ny, nz, sp, freeze=L.FREEZE_MASK, precision=L.PREC_FP64, arith=arith, tile=tile << 8) as c:
        c.load(field, frozen)
        changes = [c.sweep(sn) for sn in range(1, 9)]
        c.store(out)
    return out, changes


def spheres(shape, sp):
    w = W.random_spheres(*shape, *sp, 4, 1.5 * sp[0], 9.0 * sp[0], seed=sum(shape))
    w.field[1, 1, 1] = 0.25 * sp[0]
    return w


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("sp", SPACINGS)
def test_reference_equals_plain_solver(shape, sp):
    w = spheres(shape, sp)
    for frozen in (w.frozen, None):
        a, b = (sweeps(w.field, frozen, sp, L.ARITH_REFERENCE, t) for t in (6, 1))
        assert a[0].tobytes() == b[0].tobytes()
        assert a[1] == b[1]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("sp", SPACINGS)
def test_fast_near_plain_solver(shape, sp):
    w = spheres(shape, sp)
    a, b = (sweeps(w.field, w.frozen, sp, L.ARITH_FAST, t)[0] for t in (6, 1))
    np.testing.assert_allclose(a, b, rtol=4 * 4 * 2.0**-53 * 8 * sum(shape), atol=0)


@pytest.mark.parametrize("h", [1e-40, 1e-25, 1e-12, 1e14, 1e25, 1e40])
def test_reference_at_extreme_spacings(h):
    w = spheres((20, 13, 35), (1.0, 1.0, 1.0))
    f = np.where(w.field < 1e4, w.field * h, 1e4 * h)
    a, b = (sweeps(f, w.frozen, (h, 1.5 * h, 0.5 * h), L.ARITH_REFERENCE, t)[0] for t in (6, 1))
    assert a.tobytes() == b.tobytes()


@pytest.mark.parametrize("arith", [L.ARITH_REFERENCE, L.ARITH_FAST])
def test_odd_values(arith):
    """Random values of every kind, mixed through the grid: far apart (one term),
    equal, negative, zeros of both signs, subnormal, huge, infinite, NaN."""
    r = np.random.default_rng(7)
    f = r.uniform(0.0, 3.0, (37, 22, 19))
    odd = np.array([-1.5, 0.0, -0.0, 5e-324, 1e-300, 1e9, 1e155, 1e300, 1.7e308, np.inf, np.inf, np.nan, 2.0, 2.0])
    pick = r.random(f.shape) < 0.2
    f[pick] = r.choice(odd, pick.sum())
    frozen = (r.random(f.shape) < 0.1).astype(np.uint8)
    a, b = (sweeps(f, frozen, (1.0, 1.0, 1.0), arith, t)[0] for t in (6, 1))
    if arith == L.ARITH_REFERENCE:
        assert np.array_equal(a, b, equal_nan=True)
    else:
        assert np.array_equal(np.isfinite(a), np.isfinite(b))
        ok = np.isfinite(b)
        np.testing.assert_allclose(a[ok], b[ok], rtol=1e-12, atol=1e-12)  # values to 3, some cancelling
