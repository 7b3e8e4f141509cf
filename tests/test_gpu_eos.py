"""The equation of state at its edges."""
import numpy as np
import pytest

from oracle import Oracle
from sources_b200 import Solver, scenes
from sources_b200.abi import SPHG_FP32, SPHG_FP64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [SPHG_FP64, SPHG_FP32])
def test_infinite_density_ratio(cuda_ok, precision):
    """A water particle without volume, or of infinite density, has infinite pressure and sound speed, as
    rho / (rho0 vof) to any power; one whose power overflows has infinite pressure alone."""
    s = scenes.small("two_phase", precision=precision)
    P = s.phases[0]
    P.vof[3], P.rho[40], P.rho[77] = 0.0, np.inf, 1e50
    o = Oracle(s)
    assert o.single_step(1) == 0
    want = o.download(1)
    with Solver(s) as g:
        g.single_step(1)
        got = g.download(1)
    for i in (3, 40, 77):
        assert np.isposinf(want.p[i]) and np.isposinf(got.p[i]), (i, got.p[i])
    for i in (3, 40):
        assert np.isposinf(want.c[i]) and np.isposinf(got.c[i]), (i, got.c[i])
    assert abs(got.c[77] - want.c[77]) <= 4 * 2.0 ** -52 * want.c[77]


def test_fp64_pressure_is_the_references(cuda_ok):
    """FP64: pow, as the reference and the oracle call it.  Both are within two ulp of the power, so the pressures
    differ by four at most (b times the power; p itself may be much smaller)."""
    s = scenes.small("two_phase", precision=SPHG_FP64)
    P = s.phases[0]
    P.rho *= 1 + np.random.default_rng(5).uniform(-0.02, 0.02, P.n)
    o = Oracle(s)
    assert o.single_step(1) == 0
    with Solver(s) as g:
        g.single_step(1)
        got, want = g.download(1), o.download(1)
    assert (np.abs(got.p - want.p) <= 4 * 2.0 ** -52 * (s.params.water.b + np.abs(want.p))).all()
    assert (np.abs(got.c - want.c) <= 4 * 2.0 ** -52 * want.c).all()
