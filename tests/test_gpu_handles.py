"""Contexts take their stream, events and pinned block from a pool shared by the
process's threads: solves that overlap on several threads, hand sets over to one
another and have the pool emptied under them give the bits of a lone solve."""
import threading

import numpy as np
import pytest

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api
from pdfs_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_overlapping_solves_on_threads():
    w = W.random_spheres(40, 33, 50, 1.0, 1.0, 1.0, 3, 2.0, 8.0, seed=2)
    kinds = [dict(precision=L.PREC_FP32), dict(precision=L.PREC_FP64, arith=L.ARITH_REFERENCE, tol=1e-9),
             dict(precision=L.PREC_FP32_POLISH64, arith=L.ARITH_PAIR, tol=1e-5)]

    def solve(kw):
        a = w.field.copy()
        api.solve(a, (1.0, 1.0, 1.0), frozen=w.frozen, freeze=L.FREEZE_MASK, **kw)
        return a.tobytes()

    want = [solve(kw) for kw in kinds]
    bad = []

    def work(t):
        for k in range(6):
            i = (t + k) % len(kinds)
            if solve(kinds[i]) != want[i]:
                bad.append((t, k))
            if t == 0 and k % 2:
                api.release_cached(0)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
