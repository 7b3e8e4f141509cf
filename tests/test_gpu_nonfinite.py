"""Infinite and NaN fields."""
import numpy as np
import pytest

from sources_b200 import Solver
from sources_b200.abi import SPHG_FP64
from test_gpu_pairs2 import build

pytestmark = pytest.mark.gpu

def scene(kind, precision, skf, phase, field, value, squeeze):
    s = build(kind, precision, skf, (13, 17, 29), squeeze)
    P = s.phases[phase]
    i = np.argmin(((P.x[:P.ntotal] - P.x[:P.ntotal].mean(0)) ** 2).sum(1))     # well inside
    getattr(P, field)[i] = value
    return s


@pytest.mark.parametrize("kind", ["granular_column", "two_phase"])
@pytest.mark.parametrize("skf", [1, 4])
def test_fp64_infinite_density(cuda_ok, kind, skf):
    """The reciprocal of an infinite mean density is zero: the particle has no XSPH velocity, and no NaN."""
    s = scene(kind, SPHG_FP64, skf, 0, "rho", np.inf, 1.0)
    i = int(np.flatnonzero(np.isinf(s.phases[0].rho))[0])
    with Solver(s) as g:
        g.single_step(1)
        assert np.abs(g.download(1).av[i]).max() <= 1e-100
