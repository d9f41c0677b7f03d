"""Device memory of a context (host code on a fake CUDA runtime, no GPU): what a context
takes beside its fields, and what happens where the bricks' mailboxes do not fit.  They
are a block of their own, left out or given back when the device is full, so that a grid
never fails for them; the fields, the frozen bits, the scheduler's words and the stage of
host transfers are what a context cannot do without."""
import re

import pytest

import fakecuda
from pdfs_gb300 import _lib as L

GRID = (320, 288, 352)
NODES = 320 * 288 * 352
KINDS = [dict(precision=L.PREC_FP64), dict(precision=L.PREC_FP64, arith=L.ARITH_FAST),
         dict(precision=L.PREC_FP64, arith=L.ARITH_PAIR), dict(precision=L.PREC_FP32),
         dict(precision=L.PREC_FP32_POLISH64, arith=L.ARITH_PAIR, scheduler=L.SCHED_OCTANT),
         dict(precision=L.PREC_FP32_POLISH64, arith=L.ARITH_PAIR, tile=9 | 5 << 8)]

SOLVE = """
kw = %r
nx, ny, nz = %r
f = np.full((nz + 2, ny + 2, nx + 2), 1e10)
with api.Context(nx, ny, nz, (1.0, 1.0, 1.0), max_sweeps=16, **kw) as c:
    c.load(f)
    c.run()
    c.store(f)
print("ok")
"""


def taken(log):
    return [int(w[1]) for w in log if w[0] == "malloc"]


def mail_of_bricks(log):
    """The last template argument (MAIL) of the brick kernels launched."""
    return {re.search(r"Lb([01])EEEv", w[1]).group(1) == "1" for w in log
            if w[0] == "launch" and "t3_sweep_kernel" in w[1]}


@pytest.mark.parametrize("kw", KINDS)
def test_mailboxes_give_way(kw):
    text, log = fakecuda.run(SOLVE % (kw, GRID))
    assert text.split() == ["ok"]
    arena, mail, stage = taken(log)
    # 16 bytes a node of 64-bit fields and 4 of FP32 ones, rows padded by up to a tenth,
    # and below 1.2 bytes of everything else
    fields = {L.PREC_FP64: 16, L.PREC_FP32: 12, L.PREC_FP32_POLISH64: 20}[kw["precision"]]
    assert arena < (fields * 1.1 + 1.2) * NODES
    assert mail <= 5.2 * NODES
    assert mail_of_bricks(log) == {True}
    # no room for the mailboxes at the start; none for the stage with them; just enough
    for room in (arena + stage, arena + max(mail, stage) + 1000, arena + mail + stage):
        text, log = fakecuda.run(SOLVE % (kw, GRID), memory=room)
        assert text.split() == ["ok"], room
    # without mailboxes bricks run, and pencils do not
    text, log = fakecuda.run(SOLVE % (kw, GRID), memory=arena + stage)
    assert mail_of_bricks(log) == {False}
    assert not any("pc_sweep_kernel" in w[1] for w in log if w[0] == "launch")
    # a device without room for the stage has none
    text, log = fakecuda.run("""
try:
    exec(%r)
except api.PdfsError as e:
    print("error", e.status)
""" % (SOLVE % (kw, GRID)), memory=arena + stage - 4096)
    assert text.split() == ["error", "-2"]


def test_batch_contexts_own_no_brick_mail():
    """A batch's rounds run on pencils: their mailboxes, and no bricks'."""
    text, log = fakecuda.run("""
f = [np.full((102, 90, 122), 1e10) for _ in range(2)]
api.solve_batch(f, [(1.0, 1.0, 1.0)] * 2, precision=L.PREC_FP64)
print("ok")
""")
    assert text.split() == ["ok"]
    mail = (120 + 15) // 16 * ((88 + 15) // 16) * 2 * (100 + 15) * 16 * 2 * 8  # two faces of 16 values a level
    assert taken(log).count(mail) == 2 and len(taken(log)) == 7  # arena, mail and stage of each, and the batch's own
    assert not any("t3_sweep_kernel" in w[1] for w in log if w[0] == "launch")
