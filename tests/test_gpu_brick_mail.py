"""Bricks hand their downwind faces over by mail, level by level (tile3d.cuh).
A whole cycle of 8 orderings in one launch (the FP32 full round, where bricks
of several sweeps run at once) against the same 8 sweeps one launch each on the
column kernel: the same bits, at the shapes where the hand-over can go wrong
-- one node past a brick, one short of it, one brick thick, several bricks --
for both spacing kinds, with and without frozen nodes, and with spacings so
small that the local solver's discriminants are subnormal floats."""
import numpy as np
import pytest

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api
from pdfs_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (16, 16, 32), (17, 16, 33), (15, 31, 31), (16, 1, 65), (33, 50, 8), (50, 43, 52), (97, 33, 64)]


def full_round(w, sp, frozen):
    """The first FP32 cycle as one launch: stop the solve after its 8 sweeps."""
    kw = dict(freeze=L.FREEZE_MASK, precision=L.PREC_FP32)
    out = np.empty_like(w.field)
    with api.Context(w.nx, w.ny, w.nz, sp, scheduler=L.SCHED_OCTANT, max_sweeps=8, **kw) as c:
        c.load(w.field, frozen)
        try:
            c.run()
        except api.PdfsError as e:
            assert e.status == L.PDFS_ERR_NOT_CONVERGED
        c.store(out)
    return out


def sequential(w, sp, frozen):
    out = np.empty_like(w.field)
    with api.Context(w.nx, w.ny, w.nz, sp, freeze=L.FREEZE_MASK, precision=L.PREC_FP32, tile=4) as c:
        c.load(w.field, frozen)
        for sn in range(1, 9):
            c.sweep(sn)
        c.store(out)
    return out


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("sp", [(1.0, 1.0, 1.0), (0.7, 1.0, 0.5)])
def test_full_round_equals_column_sweeps(shape, sp):
    w = W.random_spheres(*shape, *sp, 4, 1.5, 9.0, seed=sum(shape))
    w.field[1, 1, 1] = 0.25  # something to spread from, whatever the spheres hit
    for frozen in (w.frozen, None):
        assert full_round(w, sp, frozen).tobytes() == sequential(w, sp, frozen).tobytes()


@pytest.mark.parametrize("h", [1e-18, 1e-12, 1e14])
def test_full_round_at_extreme_spacings(h):
    sp = (h, h, h)
    w = W.random_spheres(35, 20, 40, *sp, 3, 2 * h, 8 * h, seed=5)
    assert full_round(w, sp, w.frozen).tobytes() == sequential(w, sp, w.frozen).tobytes()


@pytest.mark.parametrize("tile", [5, 7, 8])
@pytest.mark.parametrize("shape", [(17, 9, 33), (33, 24, 40), (40, 23, 70)])
def test_pair_polish_on_every_brick_shape(shape, tile):
    """The pair polish on each brick shape (16 and 8 rows, 16 and 32 planes),
    unscheduled: the same bits whatever the bricks."""
    w = W.random_spheres(*shape, 1.0, 1.0, 1.0, 3, 2.0, 8.0, seed=sum(shape))
    sp = (1.0, 1.0, 1.0)
    out = []
    for t in (9 | (5 << 8), 9 | (tile << 8)):
        a = w.field.copy()
        api.solve(a, sp, frozen=w.frozen, freeze=L.FREEZE_MASK, precision=L.PREC_FP32_POLISH64, arith=L.ARITH_PAIR,
                  tol=1e-5, tile=t)
        out.append(a)
    assert out[0].tobytes() == out[1].tobytes()
