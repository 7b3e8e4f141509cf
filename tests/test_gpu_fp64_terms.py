"""The FP64 passes' pair terms against the oracle, closer than the parity tests
look.  The passes may differ from the serial order in the order of a sum and by
contracted multiply-adds only.  For a sum of N terms t that is N + 4 rounding
errors of random sign, each at most 2^-53 of a partial sum, and a partial sum
of terms of random sign is about their root sum of squares: the bar is four
times that, taken as the mean square over the phase's particles."""
import numpy as np
import pytest

from oracle import Oracle
from sources_b200 import Solver, scenes
from sources_b200.abi import SPHG_FP64
from test_gpu_tail import radial

pytestmark = pytest.mark.gpu


# eight lanes per particle, four, and one
@pytest.mark.parametrize("n", [2500, 14000, 40000])
@pytest.mark.parametrize("skf", [1, 2, 3, 4])
@pytest.mark.parametrize("kind", ["granular_column", "two_phase"])
def test_sums_are_the_oracles_to_rounding(cuda_ok, kind, skf, n):
    dx, g = 0.0037, np.random.default_rng(n + skf)
    if kind == "two_phase":
        h = int((n * 0.3) ** 0.5)
        s = scenes.two_phase(n // h * dx, 1.25 * h * dx, n // h // 2 * dx, h // 2 * dx, h * dx, dx, skf=skf, precision=SPHG_FP64)
    else:
        w = int(n ** 0.5)
        s = scenes.granular_column(w * dx, w * dx, 2 * w * dx, 1.4 * w * dx, dx, skf, precision=SPHG_FP64)
    for P in s.phases:
        P.x[:P.ntotal] += g.normal(0, 0.06 * dx, (P.ntotal, 2))
        P.vx[:P.ntotal] = g.normal(0, 0.3, (P.ntotal, 2))
    s.params.artificial_density = 0      # drho is then one sum
    s.params.max_interaction *= 4
    o = Oracle(s)
    assert o.single_step(1) == 0
    with Solver(s) as dev:
        dev.single_step(1)
        for k, S in enumerate(s.phases):
            A, B = dev.download(k + 1), o.download(k + 1)
            a, b = (p.astype(np.int64) - 1 for p in o.pairs(k))
            i, j = np.concatenate([a, b]), np.concatenate([b, a])
            hs = float(S.hsml[0])
            d, u = S.x[i] - S.x[j], S.vx[i] - S.vx[j]
            r = np.linalg.norm(d, axis=1)
            w, dw = radial(skf, r / hs, hs)
            eps = np.where(S.itype > 0, s.params.epsilon, 1.0)[i]
            m = S.mass[j]
            terms = {"drho": m * dw / r * np.abs((u * d).sum(1)),
                     "av": eps * 2 * m / (S.rho[i] + S.rho[j]) * w * np.linalg.norm(u, axis=1)}
            cnt = np.bincount(i, minlength=S.n) + 4
            for f, t in terms.items():
                tol = 4 * 2.0 ** -53 * np.sqrt((cnt * np.bincount(i, weights=t * t, minlength=S.n)).mean())
                e = getattr(A, f) - getattr(B, f)
                rms = np.sqrt((e ** 2).reshape(S.n, -1).sum(1).mean())
                assert rms <= tol, (k + 1, f, rms / tol)
