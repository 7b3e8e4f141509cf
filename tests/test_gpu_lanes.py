"""FP64 passes with several lanes per particle (small phases): every number of
lanes against the oracle, at sizes that leave the last block partly empty and on
both sides of the rule's two lines.  The bar is the FP64 bar of the one-lane
passes: 1e-9 of the field after one right-hand side, pair sets equal."""
import numpy as np
import pytest

from oracle import Oracle
from sources_b200 import Solver, scenes
from sources_b200.abi import SPHG_FP64

pytestmark = pytest.mark.gpu

FIELDS = ("drho", "dvx", "av", "p", "rho", "dvof", "vof2", "dsxx", "dsxy", "dsyy", "dp", "vcc")


def scene(kind, n, skf):
    dx = 0.004
    if kind == "two_phase":
        h = max(6, int((n * 0.3) ** 0.5))
        s = scenes.two_phase(n // h * dx, 1.2 * h * dx, n // h // 2 * dx, h // 2 * dx, h * dx, dx, skf=skf, precision=SPHG_FP64,
                             forchheimer_b=4e4 if skf == 4 else 0.0)
    else:
        w = max(3, int(n ** 0.5))
        make = scenes.dam_break if kind == "dam_break" else scenes.granular_column
        s = make(w * dx, n // w * dx, 2 * w * dx, 1.2 * n // w * dx, dx, skf, precision=SPHG_FP64)
    s = scenes.jitter(s, 0.1 * dx, seed=n)
    for P in s.phases:
        P.vx[:P.ntotal] = np.random.default_rng(3).normal(0, 0.1, size=(P.ntotal, 2))
    return s


# 8, 8, 4, 4 and 1 lanes
@pytest.mark.parametrize("n", [40, 5003, 11027, 27001, 33013])
@pytest.mark.parametrize("kind,skf", [("dam_break", 1), ("granular_column", 4), ("two_phase", 1), ("two_phase", 4)])
def test_lanes_match_oracle(cuda_ok, kind, skf, n):
    s = scene(kind, n, skf)
    o = Oracle(s)
    assert o.single_step(1) == 0
    with Solver(s) as g:
        g.single_step(1)
        st = g.stats()
        for w in range(1 if len(s.phases) == 1 else 3):
            assert st.niac[w] == len(o.pairs(w)[0])
        for k in range(len(s.phases)):
            a, b = g.download(k + 1), o.download(k + 1)
            for f in FIELDS:
                x, y = getattr(a, f), getattr(b, f)
                assert np.abs(x - y).max() <= 1e-9 * max(np.abs(y).max(), 1e-30), (k + 1, f)
            assert np.array_equal(a.fail, b.fail)
