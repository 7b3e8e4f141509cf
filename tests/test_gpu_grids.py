"""The cell list's scan on both sides of each of its lines: chunks of 2,048 cells,
the direct sum up to 16,384 cells, the chunk sums scanned by a launch of their own
above 4,096 chunks.  A longer grid leaves every particle in the same row and
the same column, so neighbours, their order and every sum stay the same: the
states are compared bit for bit."""
import math

import numpy as np
import pytest

from sources_b200 import Solver, scenes
from sources_b200.abi import SPHG_FP32, SPHG_FP64

pytestmark = pytest.mark.gpu

ROWS = 16


def column(precision, columns):
    """A soil column in a grid of ROWS x columns cells (8 columns per support radius)."""
    s = scenes.granular_column(30 * 0.002, 20 * 0.002, 70 * 0.002, 0.05, 0.002, precision=precision)
    s = scenes.jitter(s, 2e-4, seed=4)
    p, cell = s.params, 2 * float(s.phases[0].hsml[0]) * (1 + 1e-6)
    p.y_max = p.y_min + (ROWS - 1.5) * cell
    p.x_max = p.x_min + (columns - 1.5) * cell / 8
    ncell = (math.ceil((p.x_max - p.x_min) / (cell / 8)) + 1) * (math.ceil((p.y_max - p.y_min) / cell) + 1)
    assert ncell == ROWS * columns
    return s


def state(precision, columns):
    with Solver(column(precision, columns)) as g:
        g.set_tuning(1.0, 3, 8)
        g.time_integration(5)
        st = g.stats()
        assert st.n_out_of_domain == 0
        return g.download(1), list(st.niac)


@pytest.mark.parametrize("precision", [SPHG_FP64, SPHG_FP32])
def test_longer_grids_change_nothing(cuda_ok, precision):
    want, niac = state(precision, 700)
    chunk, direct, sums = (n // ROWS for n in (2048, 16 * 1024, 4096 * 2048))
    for columns in (6 * chunk, direct - 1, direct, direct + 1, 9 * chunk, sums - 1, sums, sums + 1, sums + 65 * chunk + 5, 4 * sums + 3):
        got, n = state(precision, columns)
        assert n == niac, columns
        for f in ("x", "vx", "rho", "p", "sxx", "drho", "dvx"):
            assert np.array_equal(getattr(got, f), getattr(want, f)), (columns, f)
