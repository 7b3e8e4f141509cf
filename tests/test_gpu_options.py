"""What a step leaves in the arrays of the step before, per option."""
import numpy as np
import pytest

from oracle import Oracle
from sources_b200 import Solver, scenes
from sources_b200.abi import SPHG_FP32, SPHG_FP64

pytestmark = pytest.mark.gpu


# 480 and 40,000 particles: several lanes per particle and one, in FP64
@pytest.mark.parametrize("cells", [(10, 20, 40), (200, 180, 220)])
@pytest.mark.parametrize("precision", [SPHG_FP64, SPHG_FP32])
@pytest.mark.parametrize("summed", [0, 1])
def test_density_before_the_step(cuda_ok, precision, summed, cells):
    """rho_min is the density before the predictor, and stays the host's when the
    density is summed and never integrated (first_half, declarations_sph.f90:643)."""
    w, h, box = (n * 0.005 for n in cells)
    s = scenes.jitter(scenes.dam_break(w, h, box, 1.2 * h, 0.005, precision=precision), 5e-4, seed=2)
    s.params.summation_density = summed
    P = s.phases[0]
    P.rho_min[:] = np.arange(P.n) + 0.5
    o = Oracle(s)
    with Solver(s) as g:
        for steps in (1, 2):
            assert o.time_integration(steps) == 0
            g.time_integration(steps)
            got = g.download(1)
            if summed:
                assert np.array_equal(got.rho_min, P.rho_min)
            elif steps == 2:
                assert not np.array_equal(got.rho_min, P.rho_min)
            want = o.download(1).rho_min
            tol = 1e-9 if precision == SPHG_FP64 else 5e-6     # the density's bars of the parity tests
            assert np.abs(got.rho_min - want).max() <= tol * np.abs(want).max(), steps
