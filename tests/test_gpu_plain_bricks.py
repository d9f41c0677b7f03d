"""The pencil tiles' plain sweeps on bricks (tile3d_plain.cu) against the other
kernels: FP32 against the columns, pairs and mixed against the selectable brick
tile (whose single sweeps are the masked kernel's), the same bits after each of the
8 orderings -- at one node past a brick, one short of it, one brick thick, several
bricks -- for both spacing kinds, with and without frozen nodes, and through the
replace-update of a polish."""
import numpy as np
import pytest

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api
from pdfs_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (8, 8, 32), (9, 8, 33), (7, 15, 31), (16, 16, 32), (17, 16, 33), (15, 31, 31), (16, 1, 65),
          (33, 50, 8), (50, 43, 52), (97, 33, 64)]
SPACINGS = [(1.0, 1.0, 1.0), (0.7, 1.0, 0.5)]


def sweeps(w, sp, frozen, **kw):
    out, changes = np.empty_like(w.field), []
    with api.Context(w.nx, w.ny, w.nz, sp, freeze=L.FREEZE_MASK, **kw) as c:
        c.load(w.field, frozen)
        changes = [c.sweep(sn) for sn in range(1, 9)]
        c.store(out)
    return out.tobytes(), changes


def field(shape, sp):
    w = W.random_spheres(*shape, *sp, 4, 1.5, 9.0, seed=sum(shape))
    w.field[1, 1, 1] = 0.25  # something to spread from, whatever the spheres hit
    return w


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("sp", SPACINGS)
def test_fp32_sweeps_equal_column_sweeps(shape, sp):
    w = field(shape, sp)
    for frozen in (w.frozen, None):
        a, b = (sweeps(w, sp, frozen, precision=L.PREC_FP32, tile=t) for t in (10, 4))
        assert a[0] == b[0]
        assert a[1] == pytest.approx(b[1], rel=1e-6)  # the change of a node, in either kernel's rounding


def test_fp32_sweeps_of_wide_levels():
    """A grid past the level width of the small bricks (37000 nodes a level)."""
    w = field((347, 323, 329), (1.0, 1.0, 1.0))
    a, b = (sweeps(w, (1.0, 1.0, 1.0), w.frozen, precision=L.PREC_FP32, tile=t) for t in (10, 4))
    assert a[0] == b[0]


@pytest.mark.parametrize("arith", [L.ARITH_PAIR, L.ARITH_MIXED])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("sp", SPACINGS)
def test_pair_and_mixed_sweeps_equal_brick_tile(arith, shape, sp):
    w = field(shape, sp)
    for frozen in (w.frozen, None):
        a, b = (sweeps(w, sp, frozen, precision=L.PREC_FP64, arith=arith, tile=t << 8) for t in (6, 5))
        assert a[0] == b[0]
        assert a[1] == pytest.approx(b[1], rel=1e-6)


@pytest.mark.parametrize("arith", [L.ARITH_PAIR, L.ARITH_MIXED])
@pytest.mark.parametrize("shape", [(17, 9, 33), (33, 24, 40), (40, 23, 70)])
def test_polish_equals_brick_tile(arith, shape):
    w = W.random_spheres(*shape, 1.0, 1.0, 1.0, 3, 2.0, 8.0, seed=sum(shape))
    out = []
    for t in (6, 5):
        a = w.field.copy()
        st = api.solve(a, (1.0, 1.0, 1.0), frozen=w.frozen, freeze=L.FREEZE_MASK, precision=L.PREC_FP32_POLISH64,
                       arith=arith, tol=1e-5, tile=10 | (t << 8))
        out.append((a.tobytes(), st["sweeps_fp64"]))
    assert out[0] == out[1]
