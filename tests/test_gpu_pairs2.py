"""The FP32 pair passes with two particles per lane pair (sphg_pairs2.cuh) at
the shapes where they can go wrong: blocks that span several rows of cells
(read through L1 instead of shared memory), particles paired across rows, odd
particle counts, and crowds with more candidates than the hit masks hold.

The reference is the FP64 path, which the oracle pins (test_gpu_parity.py).  The
pair counts must be equal.  drho and dvx are held to a bound derived from the
terms themselves: every FP32 operand carries a relative error of 2^-24, so a
sum of N terms is off by at most (N + 32) 2^-24 times the sum of the terms'
magnitudes (operands counted by their own size, not their difference's)."""
import numpy as np
import pytest

from sources_b200 import Solver, scenes
from sources_b200.abi import SPHG_FP32, SPHG_FP64, SPHG_SOIL

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def build(kind, precision, skf, cells, squeeze):
    w, h, box = cells
    dx = 0.005
    if kind == "granular_column":
        s = scenes.granular_column(w * dx, h * dx, box * dx, 1.2 * h * dx, dx, skf, precision=precision)
    else:
        s = scenes.two_phase(box * dx, 1.2 * h * dx, w * dx, h // 2 * dx, h * dx, dx, skf=skf, precision=precision)
    s = scenes.jitter(s, 0.1 * dx, seed=w + h)
    g = np.random.default_rng(7)
    for P in s.phases:
        P.vx[:P.ntotal] = g.normal(0, 0.1, size=(P.ntotal, 2))
        P.x *= squeeze
    s.params.max_interaction *= 8
    return s


def radial(skf, q, h):
    """(W, |grad W|) of the kernel at q = r / h."""
    if skf == 1:
        f = 15.0 / (7.0 * np.pi * h * h)
        return (f * np.where(q <= 1, 2 / 3 - q * q + q ** 3 / 2, (2 - q) ** 3 / 6),
                f / h * np.where(q <= 1, q * (2 - 1.5 * q), (2 - q) ** 2 / 2))
    f, u = 7.0 / (4.0 * np.pi * h * h), 1 - q / 2
    return f * u ** 4 * (1 + 2 * q), f / h * 5 * q * u ** 3


def ends(g, which, swap=False):
    i, j = g.pairs(which)
    i, j = i.astype(np.int64) - 1, j.astype(np.int64) - 1
    if which == 2:
        return (j, i) if swap else (i, j)
    return np.concatenate([i, j]), np.concatenate([j, i])


def bounds(s, g, A, k):
    """Error bounds of drho and dvx of phase k from the FP64 state A."""
    P, p, skf = A[k], s.params, s.params.skf
    h, n = float(P.hsml[0]), P.n
    soil = P.material == SPHG_SOIL
    i, j = ends(g, k)
    w, dw = radial(skf, np.linalg.norm(P.x[i] - P.x[j], axis=1) / h, h)
    add = lambda v: np.bincount(i, weights=v, minlength=n)  # noqa: E731
    cnt = add(np.ones(len(i)))
    speed = np.linalg.norm(P.vx, axis=1)
    vv = speed[i] + speed[j]
    vol = P.mass / P.rho
    c = np.maximum(P.c, p.soil.c if soil else p.water.c)
    drho = add(P.mass[j] * vv * dw) + p.delta * h * c * add(vol[j] * (P.rho[i] + P.rho[j]) * 2 * dw / h * 2)
    f = np.abs(P.p) + np.abs(P.sxx) + np.abs(P.sxy) + np.abs(P.syy)
    dv = add(vol[j] * (f[i] + f[j]) * dw) / P.rho
    dv += add(P.mass[j] * p.alpha * (c[i] + c[j]) * vv / P.rho[j] * dw) + abs(p.gravity)
    if len(A) == 2:
        o = A[1 - k]
        ci, cj = ends(g, 2, swap=k == 1)
        wc, dwc = radial(skf, np.linalg.norm(P.x[ci] - o.x[cj], axis=1) / h, h)
        ovol = o.mass / o.rho
        u = speed[ci] + np.linalg.norm(o.vx, axis=1)[cj]
        fac = abs(p.numeric_gravity) / p.soil.permeability
        dv += np.bincount(ci, weights=fac * ovol[cj] * wc * u + ovol[cj] * np.abs(o.p[cj]) * dwc / P.rho[ci], minlength=n)
        cnt = cnt + np.bincount(ci, minlength=n)
        r = np.linalg.norm(P.x[i] - P.x[j], axis=1)
        z = P.dspp / r
        dv += add(np.where(r <= P.dspp, 64 * p.dd * (z ** p.p1 + z ** p.p2) / r, 0.0))   # powers: 16x each operand's error
    return (cnt + 32) * EPS * drho, (cnt + 32) * EPS * dv


# (column or block width, height, box width) in cells: rows of 24 particles (a block of 128 spans six rows), an ordinary
# box, and rows longer than a block; squeeze < 1 crowds the particles
@pytest.mark.parametrize("squeeze", [1.0, 0.6, 0.4])
@pytest.mark.parametrize("cells", [(3, 31, 6), (13, 17, 29), (90, 9, 190)])
@pytest.mark.parametrize("skf", [1, 4])
@pytest.mark.parametrize("kind", ["granular_column", "two_phase"])
def test_paired_passes_match_fp64(cuda_ok, kind, skf, cells, squeeze):
    s64, s32 = (build(kind, prec, skf, cells, squeeze) for prec in (SPHG_FP64, SPHG_FP32))
    with Solver(s64) as a, Solver(s32) as b:
        a.single_step(1)
        b.single_step(1)
        sa, sb = a.stats(), b.stats()
        for f in ("niac", "maxiac", "miniac", "noiac"):
            assert list(getattr(sa, f)) == list(getattr(sb, f)), f
        A = [a.download(k + 1) for k in range(len(s64.phases))]
        for k in range(len(A)):
            B = b.download(k + 1)
            for f, tol in zip(("drho", "dvx"), bounds(s64, a, A, k)):
                e = np.abs(getattr(B, f) - getattr(A[k], f)).reshape(B.n, -1).max(1)
                bad = np.flatnonzero(~(e <= tol))
                assert bad.size == 0, (k + 1, f, bad.size, B.n, float((e / tol).max()))


@pytest.mark.parametrize("drop", [0, 1, 2, 3])
def test_odd_particle_counts(cuda_ok, drop):
    """n, n-1, .. particles: the last lane pair is whole or half, in the last
    block alone or not; the state after six steps (predictor and corrector)
    agrees with FP64 to the FP32 budget of the 30-step test."""
    def cut(precision):
        s = build("granular_column", precision, 1, (13, 17, 29), 1.0)
        P = s.phases[0]
        keep = P.n - P.n % 128 + 1 - drop     # 1 particle in the last block, then 128, 127, 126
        Q = type(P)(keep, P.ntotal, P.material, P.dspp)
        for f in ("x", "vx", "rho", "p", "c", "mass", "hsml", "vof", "sxx", "sxy", "syy", "itype"):
            getattr(Q, f)[...] = getattr(P, f)[:keep]
        s.phases = [Q]
        return s
    s64, s32 = cut(SPHG_FP64), cut(SPHG_FP32)
    with Solver(s64) as a, Solver(s32) as b:
        a.time_integration(6)
        b.time_integration(6)
        assert list(a.stats().niac) == list(b.stats().niac)
        A, B = a.download(1), b.download(1)
        for f, tol in (("x", 5e-7), ("vx", 5e-4), ("rho", 5e-6)):
            x, y = getattr(A, f), getattr(B, f)
            assert np.abs(x - y).max() <= tol * np.abs(x).max(), f


@pytest.mark.parametrize("kind", ["granular_column", "two_phase"])
def test_coincident_particles_without_etq(cuda_ok, kind):
    """etq = 0 leaves the viscous denominator r^2 alone: a particle's own slot
    and coincident neighbours (r = 0) add nothing."""
    s64, s32 = (build(kind, prec, 1, (13, 17, 29), 1.0) for prec in (SPHG_FP64, SPHG_FP32))
    for s in (s64, s32):
        s.params.etq = 0.0
        for P in s.phases:
            P.x[7] = P.x[6]
            P.vx[7] = P.vx[6] + 0.05
    with Solver(s64) as a, Solver(s32) as b:
        a.single_step(1)
        b.single_step(1)
        assert list(a.stats().niac) == list(b.stats().niac)
        for k, P in enumerate(s64.phases):
            A, B = a.download(k + 1), b.download(k + 1)
            for f in ("drho", "dvx", "av"):
                x, y = getattr(A, f), getattr(B, f)
                assert np.isfinite(x).all() and np.isfinite(y).all(), f
                assert np.abs(x - y).max() <= 2e-3 * np.abs(x).max(), f   # the FP32 budget of one step's rates
