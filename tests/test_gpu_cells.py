"""The cell list: its scan on both sides of its lines (chunks of 2,048 cells, the
direct sum up to 65,536), and cells ordered by the gather or by the sort.  A
step that reorders the state takes the sort, one that does not the gather; the
neighbours, their order and every sum are the same, so the states are compared
bit for bit."""
import numpy as np
import pytest

from sources_b200 import Solver, scenes
from sources_b200.abi import SPHG_FP32, SPHG_FP64

pytestmark = pytest.mark.gpu


def column(precision, span):
    """A soil column in a grid that reaches span times its box to the right, with a crowd of 60 particles in one cell."""
    s = scenes.granular_column(30 * 0.002, 20 * 0.002, 70 * 0.002, 0.05, 0.002, precision=precision)
    s = scenes.jitter(s, 2e-4, seed=4)
    P, g = s.phases[0], np.random.default_rng(9)
    P.x[100:160] = P.x[100] + g.uniform(-1e-4, 1e-4, size=(60, 2))
    perm = g.permutation(P.ntotal)       # original indices in no spatial order
    P.x[:P.ntotal] = P.x[:P.ntotal][perm]
    s.params.x_max = s.params.x_min + span * (s.params.x_max - s.params.x_min)
    s.params.max_interaction *= 16
    s.params.dt *= 0.01                  # the crowd must not fly apart
    return s


# from a few thousand cells to several times 10,000 at 8 per support radius; few at whole cells
@pytest.mark.parametrize("span,split", [(0.5, 8), (1, 8), (8, 8), (21, 8), (30, 8), (4, 1)])
@pytest.mark.parametrize("precision", [SPHG_FP64, SPHG_FP32])
def test_sort_and_gather_give_the_same_order(cuda_ok, precision, span, split):
    s = column(precision, span)
    got = []
    for interval in (0, 1, 3):           # never, always and sometimes reordering
        with Solver(s) as g:
            g.set_tuning(1.0, interval, split)
            g.time_integration(7)
            got.append((g.download(1), list(g.stats().niac), g.stats().n_out_of_domain))
    for P, niac, out in got[1:]:
        assert niac == got[0][1] and out == got[0][2]
        for f in ("x", "vx", "rho", "p", "sxx", "drho", "dvx", "itype"):
            assert np.array_equal(getattr(P, f), getattr(got[0][0], f)), f
    if span < 1:
        assert got[0][2] > 0             # clamped particles counted, each step anew
    s64 = column(SPHG_FP64, span)
    with Solver(s64) as g:
        g.set_tuning(1.0, 3, split)
        g.time_integration(7)
        i, j = g.pairs(0)
        Q = g.download(1)
    d = Q.x[:, None, :] - Q.x[None, :, :]
    r = 2 * Q.hsml[0]
    want = np.argwhere(np.triu(np.sqrt(d[..., 0] ** 2 + d[..., 1] ** 2) < r, 1))
    assert np.array_equal(np.stack([i, j], 1) - 1, want)


def test_counters_across_kinds_of_steps(cuda_ok):
    """Right-hand sides, steps, new positions and statistics in any order: each step's counters are its own."""
    s = column(SPHG_FP64, 0.5)
    with Solver(s) as g:
        g.time_integration(3)
        a = g.stats()
        for _ in range(3):
            g.single_step(5)
            b = g.stats()
            assert list(b.niac) == list(g.stats().niac)
            g.time_integration(1)
            c = g.stats()
            assert c.n_out_of_domain == a.n_out_of_domain == b.n_out_of_domain
            assert 0 < c.maxiac[0] < 2 * a.maxiac[0] and abs(c.niac[0] - a.niac[0]) < 0.01 * a.niac[0]
            g.upload(1, g.download(1))
            g.time_integration(2)
            d = g.stats()
            assert d.n_out_of_domain == a.n_out_of_domain and abs(d.niac[0] - a.niac[0]) < 0.01 * a.niac[0]
