"""A particle with an infinite or NaN field spoils its neighbours' sums and no
others': the FP32 paired passes, which look at a candidate for two particles at
once, against the FP64 passes, which visit one particle's neighbours only."""
import numpy as np
import pytest

from sources_b200 import Solver
from sources_b200.abi import SPHG_FP32, SPHG_FP64
from test_gpu_pairs2 import build

pytestmark = pytest.mark.gpu

FIELDS = ("drho", "dvx", "av", "dvof", "vof2", "dsxx", "dsxy", "dsyy", "dp", "vcc")


def scene(kind, precision, skf, phase, field, value, squeeze):
    s = build(kind, precision, skf, (13, 17, 29), squeeze)
    P = s.phases[phase]
    i = np.argmin(((P.x[:P.ntotal] - P.x[:P.ntotal].mean(0)) ** 2).sum(1))     # well inside
    getattr(P, field)[i] = value
    return s


CASES = [("granular_column", 0, "vx", np.nan), ("granular_column", 0, "vx", np.inf), ("granular_column", 0, "p", np.inf),
         ("granular_column", 0, "rho", np.inf), ("two_phase", 0, "vx", np.nan), ("two_phase", 0, "vx", -np.inf),
         ("two_phase", 0, "rho", np.inf), ("two_phase", 1, "vx", np.nan), ("two_phase", 1, "p", np.inf),
         ("two_phase", 1, "rho", np.nan), ("two_phase", 1, "rho", np.inf)]


@pytest.mark.parametrize("kind", ["granular_column", "two_phase"])
@pytest.mark.parametrize("skf", [1, 4])
def test_fp64_infinite_density(cuda_ok, kind, skf):
    """The reciprocal of an infinite mean density is zero: the particle has no XSPH velocity, and no NaN."""
    s = scene(kind, SPHG_FP64, skf, 0, "rho", np.inf, 1.0)
    i = int(np.flatnonzero(np.isinf(s.phases[0].rho))[0])
    with Solver(s) as g:
        g.single_step(1)
        assert np.abs(g.download(1).av[i]).max() <= 1e-100


# squeeze 0.4: pairs with more candidates than the masks hold, visited in two parts
@pytest.mark.parametrize("squeeze", [1.0, 0.4])
@pytest.mark.parametrize("skf", [1, 2, 3, 4])
@pytest.mark.parametrize("kind,phase,field,value", CASES)
def test_only_neighbours_are_spoilt(cuda_ok, kind, phase, field, value, skf, squeeze):
    s64, s32 = (scene(kind, prec, skf, phase, field, value, squeeze) for prec in (SPHG_FP64, SPHG_FP32))
    with Solver(s64) as a, Solver(s32) as b:
        a.single_step(1)
        b.single_step(1)
        assert list(a.stats().niac) == list(b.stats().niac)
        spoilt = 0
        for k in range(len(s64.phases)):
            A, B = a.download(k + 1), b.download(k + 1)
            for f in FIELDS:
                x, y = (np.isfinite(getattr(Q, f)).reshape(Q.n, -1).all(1) for Q in (A, B))
                assert np.array_equal(x, y), (k + 1, f, int((x & ~y).sum()), int((y & ~x).sum()), int((~x).sum()))
                spoilt += int((~x).sum())
                u, v = getattr(A, f)[x], getattr(B, f)[x]
                if u.size:
                    assert np.abs(u - v).max() <= 2e-3 * np.abs(u).max() + 1e-30, (k + 1, f)   # the FP32 budget of one step's rates
        assert spoilt > 0
