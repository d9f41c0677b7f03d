"""Bricks without mailboxes (contexts whose device had no room for them; here a test
hook asks for it) wait for whole upwind bricks: the bits of the same sweeps with mail --
plain, masked and recording sweeps, octant rounds and whole solves, on every brick tile
and on the default ones, at one node past a brick, one short of it, one brick thick and
several bricks -- and a brick that hands nothing over ends in the bounded wait's error."""
import numpy as np
import pytest

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api
from pdfs_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (17, 16, 33), (15, 31, 31), (16, 1, 65), (33, 50, 8), (50, 43, 52), (97, 33, 64)]
HOOK = "PDFS_TEST_NO_BRICK_MAIL"
KINDS = [dict(precision=L.PREC_FP32, tile=t) for t in (0, 8, 9, 11)] + \
    [dict(precision=L.PREC_FP64, arith=a, tile=t << 8) for a in (L.ARITH_REFERENCE, L.ARITH_FAST, L.ARITH_MIXED,
                                                                 L.ARITH_PAIR) for t in (0, 5, 7, 8)]


def field(shape):
    w = W.random_spheres(*shape, 1.0, 1.0, 1.0, 4, 1.5, 9.0, seed=sum(shape))
    w.field[1, 1, 1] = 0.25
    return w


def both(monkeypatch, f):
    a = f()
    monkeypatch.setenv(HOOK, "1")
    b = f()
    monkeypatch.delenv(HOOK)
    return a, b


def sweeps(w, sp, kw):
    """The 8 orderings: three plain, two that record block changes, three masked."""
    out, rec = np.empty_like(w.field), []
    r = np.random.default_rng(1)
    with api.Context(w.nx, w.ny, w.nz, sp, freeze=L.FREEZE_MASK, **kw) as c:
        c.load(w.field, w.frozen)
        nb = c.blocks()[::-1]
        for sn in range(1, 9):
            chg = np.zeros(nb, np.float32)
            act = (r.random(nb) < 0.6).astype(np.uint8)
            rec.append(c.sweep(sn, active=act if sn > 5 else None, block_change=chg if sn > 3 else None))
            rec.append(chg.tobytes())
        c.store(out)
    return out.tobytes(), rec


@pytest.mark.parametrize("kw", KINDS)
@pytest.mark.parametrize("shape", SHAPES)
def test_sweeps_without_mail(shape, kw, monkeypatch):
    w = field(shape)
    a, b = both(monkeypatch, lambda: sweeps(w, (1.0, 1.0, 1.0), kw))
    assert a[0] == b[0]
    # the plain sweeps' changes are rounded per kernel; the others' kernel is the same
    assert a[1][6:] == b[1][6:] and a[1][0:6:2] == pytest.approx(b[1][0:6:2], rel=1e-6)


@pytest.mark.parametrize("arith", [L.ARITH_REFERENCE, L.ARITH_FAST, L.ARITH_MIXED, L.ARITH_PAIR])
@pytest.mark.parametrize("sp", [(1.0, 1.0, 1.0), (0.7, 1.0, 0.5)])
@pytest.mark.parametrize("sched", [L.SCHED_OCTANT, L.SCHED_LEARNED])
def test_solves_without_mail(sched, sp, arith, monkeypatch):
    w = W.random_spheres(75, 60, 83, *sp, 6, 2.0, 9.0, seed=4)

    def solve():
        a = w.field.copy()
        st = api.solve(a, sp, frozen=w.frozen, freeze=L.FREEZE_MASK, precision=L.PREC_FP32_POLISH64, arith=arith,
                       scheduler=sched, tol=1e-5)
        return a.tobytes(), st["sweeps_fp32"], st["sweeps_fp64"], st["voxel_updates"]

    a, b = both(monkeypatch, solve)
    assert a == b


def test_wait_without_mail_times_out(monkeypatch):
    w = field((50, 43, 52))
    monkeypatch.setenv(HOOK, "1")
    monkeypatch.setenv("PDFS_TEST_POISON_COLUMN", "0")
    with api.Context(w.nx, w.ny, w.nz, (1.0, 1.0, 1.0), precision=L.PREC_FP64, wait_ms=50) as c:
        c.load(w.field)
        with pytest.raises(api.PdfsError) as e:
            c.sweep(1)
        assert e.value.status == L.PDFS_ERR_TIMEOUT
        monkeypatch.delenv("PDFS_TEST_POISON_COLUMN")
        c.load(w.field)
        c.sweep(1)
        out = np.empty_like(w.field)
        c.store(out)
    ref = w.field.copy()
    monkeypatch.delenv(HOOK)
    api.sweep(ref, (1.0, 1.0, 1.0), 1)
    assert out.tobytes() == ref.tobytes()
