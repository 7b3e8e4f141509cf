"""Downloads of pageable arrays through the library's page-locked buffers: sizes
below and above one piece (512 KB) and the threaded threshold (4 MB), several
contexts transferring from several threads at once, and buffers handed on from
context to context.  Bytes are compared, so the bound is equality."""
import threading

import numpy as np
import pytest

from sources_b200 import Solver, scenes
from sources_b200.abi import SPHG_FP64

pytestmark = pytest.mark.gpu

FIELDS = ("x", "vx", "rho", "p", "c", "mass", "hsml", "sxx", "sxy", "syy", "drho", "itype")


def column(cells, seed):
    s = scenes.granular_column(cells * 0.002, 40 * 0.002, 3 * cells * 0.002, 0.12, 0.002, precision=SPHG_FP64)
    P, g = s.phases[0], np.random.default_rng(seed)
    for f in ("vx", "drho", "sxy"):
        getattr(P, f)[...] = g.normal(size=getattr(P, f).shape)
    return s


def same(P, Q):
    for f in FIELDS:
        assert np.array_equal(getattr(P, f), getattr(Q, f)), f


# 0.4, 0.9, 3.9 and 10 MB of state
@pytest.mark.parametrize("cells", [18, 55, 280, 760])
def test_round_trip(cuda_ok, cells):
    s = column(cells, cells)
    with Solver(s) as g:
        same(s.phases[0], g.download(1))
        t = column(cells, cells + 1)
        g.upload(1, t.phases[0])
        same(t.phases[0], g.download(1))


def test_many_contexts_and_threads(cuda_ok):
    """More transfers at once than there are buffers: the rest take the direct
    copies; every context gets its own bytes."""
    work = [column(c, 100 + i) for i, c in enumerate((18, 400, 760, 300, 55, 700))]
    bad = []

    def go(s):
        try:
            for _ in range(4):
                with Solver(s) as g:
                    same(s.phases[0], g.download(1))
        except Exception as e:   # noqa: BLE001 - reported by the test's own thread
            bad.append(repr(e))
    th = [threading.Thread(target=go, args=(s,)) for s in work]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad, bad
