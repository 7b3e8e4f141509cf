"""The last lane pair of the FP32 two-phase water passes.  With an odd number
of water particles the last pair holds one particle, and the lane of the
missing one still carries every other candidate of it: pass A records that
lane's hits and pass B replays them.  The walls end below the surface here, so
that the last sorted slot is a real particle under pressure, and its sums show
every neighbour that goes missing.

The reference is the FP64 path.  A sum of N terms is off by at most (N + 32)
2^-24 times the sum of the terms' magnitudes (test_gpu_pairs2)."""
import numpy as np
import pytest

import test_gpu_pairs2 as pairs2
from sources_b200 import Solver
from sources_b200.abi import SPHG_FP32, SPHG_FP64

pytestmark = pytest.mark.gpu

radial14 = pairs2.radial


def radial(skf, q, h):
    """(W, |grad W|) of the four kernels at q = r / h."""
    if skf in (1, 4):
        return radial14(skf, q, h)
    if skf == 2:
        w = np.exp(-q * q) / (np.pi * h * h)
        return w, 2 * q / h * w
    f = 7.0 / (478.0 * np.pi * h * h)
    a, b, c = ((np.maximum(n - q, 0.0)) for n in (3, 2, 1))
    dw = np.where(q <= 1, q * np.abs(-120 + 120 * q - 50 * q * q), 5 * a ** 4 + 30 * b ** 4)
    return f * (a ** 5 + 6 * b ** 5 + 15 * c ** 5), f / h * dw


def scene(precision, skf, drop, squeeze):
    s = pairs2.build("two_phase", precision, skf, (13, 17, 29), squeeze)
    P, g = s.phases[0], np.random.default_rng(11)
    dx = 0.005 * squeeze
    real = np.arange(P.n) < P.ntotal
    keep = np.flatnonzero(real | (P.x[:, 1] < P.x[real, 1].max() - 9 * dx))
    keep = np.delete(keep, P.ntotal + np.arange(drop))
    Q = type(P)(len(keep), P.ntotal, P.material, P.dspp)
    for f in ("x", "vx", "rho", "p", "c", "mass", "hsml", "vof", "sxx", "sxy", "syy", "itype"):
        getattr(Q, f)[...] = getattr(P, f)[keep]
    Q.rho *= 1 + 0.01 * g.uniform(0.5, 1.0, Q.n)      # pressed together: p well above zero at the surface too
    s.phases[0] = Q
    return s


def water_bounds(s, g, A):
    """Error bounds of av and dvof of the water."""
    P, S, p = A[0], A[1], s.params
    h, n = float(P.hsml[0]), P.n
    i, j = pairs2.ends(g, 0)
    r = np.linalg.norm(P.x[i] - P.x[j], axis=1)
    w, dw = radial(p.skf, r / h, h)
    speed = np.linalg.norm(P.vx, axis=1)
    add = lambda v: np.bincount(i, weights=v, minlength=n)  # noqa: E731
    eps = np.where(P.itype > 0, p.epsilon, 1.0)
    av = eps * add(2 * P.mass[j] / (P.rho[i] + P.rho[j]) * w * (speed[i] + speed[j]))
    dvof = 2 * p.delta * h * P.c * add(P.mass[j] / P.rho[j] * (P.vof[i] + P.vof[j]) * dw / r)
    ci, cj = pairs2.ends(g, 2)
    dwc = radial(p.skf, np.linalg.norm(P.x[ci] - S.x[cj], axis=1) / h, h)[1]
    dvof += np.bincount(ci, weights=S.mass[cj] / p.soil.rho0 * dwc * (speed[ci] + np.linalg.norm(S.vx, axis=1)[cj]), minlength=n)
    cnt = add(np.ones(len(i))) + np.bincount(ci, minlength=n) + 32
    return cnt * pairs2.EPS * av, cnt * pairs2.EPS * dvof


# squeeze 0.25: more candidates of the last pair than the masks hold (they are tested again in pass B)
@pytest.mark.parametrize("squeeze", [1.0, 0.25])
@pytest.mark.parametrize("drop", [0, 1, 2, 3])
@pytest.mark.parametrize("skf", [1, 2, 3, 4])
def test_last_particle_keeps_every_neighbour(cuda_ok, monkeypatch, skf, drop, squeeze):
    monkeypatch.setattr(pairs2, "radial", radial)
    s64, s32 = (scene(prec, skf, drop, squeeze) for prec in (SPHG_FP64, SPHG_FP32))
    assert s64.phases[0].itype[np.argmax(s64.phases[0].x[:, 1])] > 0
    with Solver(s64) as a, Solver(s32) as b:
        a.single_step(1)
        b.single_step(1)
        assert list(a.stats().niac) == list(b.stats().niac)
        A, B = [a.download(k + 1) for k in (0, 1)], b.download(1)
        tol = dict(zip(("drho", "dvx"), pairs2.bounds(s64, a, A, 0)))
        tol.update(zip(("av", "dvof"), water_bounds(s64, a, A)))
        for f, t in tol.items():
            e = np.abs(getattr(B, f) - getattr(A[0], f)).reshape(B.n, -1).max(1)
            bad = np.flatnonzero(~(e <= t))
            assert bad.size == 0, (f, bad.size, B.n, float((e / t).max()))
