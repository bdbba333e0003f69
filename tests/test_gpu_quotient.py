"""FP64 dt / rho is the IEEE quotient whatever the sum of the two densities
looks like.  Neighbouring columns hold a usual density and one up to 2^29
times smaller, so that the sum fills up to 53 bits of a double, and dt is
chosen so that 2 dt / sum lies as near to the middle between two doubles as a
quotient by such a sum can.  One velocity update of such a plan is restated in
exact rational arithmetic, rounded operation by operation."""
import random
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def hard_case(seed, shift):
    """dt and two densities, float32 numbers whose sum is an odd multiple of
    its 2^(23 + shift)-th part: M of 54 bits, odd, with M R = +-1 modulo a power
    of two makes a / R differ from the midpoint M by 1 / (M R) of itself."""
    rng = random.Random(seed)
    while True:
        big, small = rng.randrange(1 << 23, 1 << 24), rng.randrange(1, 1 << 24, 2)
        big -= big % 2
        R = (big << shift) + small
        p = R.bit_length()
        t = p + 1
        sign = rng.choice([1, -1])
        M = -sign * pow(R, -1, 1 << t) % (1 << t)
        M += rng.randrange(1 << 53, 1 << 54) >> t << t
        if not 1 << 53 <= M < 1 << 54:
            continue
        a = (M * R + sign) >> t
        assert (a << t) == M * R + sign
        if p == 24 + shift and a.bit_length() <= 53:
            k = 2.0 ** (12 - p)   # the larger density in [2048, 4096)
            return a * 2.0 ** -62, (big << shift) * k, small * k


def rounded_vx(s, b, v, idx, idy, idz, cell):
    """vx after one update of a cell outside the layers from the stresses s
    (sxx, sxy, sxz) and the factor b, each operation rounded once."""
    k, j, i = cell
    sxx, sxy, sxz = s
    f = Fraction
    x1 = float(f(float(f(sxx[k, j, i]) - f(sxx[k, j, i - 1]))) * f(idx))
    x2 = float(f(sxy[k, j, i]) - f(sxy[k, j - 1, i]))
    x3 = float(f(sxz[k, j, i]) - f(sxz[k - 1, j, i]))
    t = float(f(x2) * f(idy) + f(x1))
    t = float(f(x3) * f(idz) + f(t))
    return float(f(b) * f(t) + f(v)), t


@pytest.mark.parametrize("shift", [0, 8, 9, 10, 11, 18, 29])
@pytest.mark.parametrize("schedule", [1, -1], ids=["two kernels", "open"])
def test_fp64_quotient_is_correctly_rounded(built, shift, schedule):
    from ela3d_gb300 import FP64, Plan, ShotParams, variants

    n = 16
    first = next(q for q, v in enumerate(variants()) if v.fp64)
    tune = {} if schedule < 0 else {"variant": first, "schedule": schedule, "chunk": 8}
    for seed in range(6):
        dt, r0, r1 = hard_case(seed, shift)
        p = ShotParams(nx=n, ny=n, nz=n, nstep=3, dt=dt, npml=0, f0=25.0, t0=2e-3, src=(8, 8, 8), src_w=(1.0, 1.0, 1.0),
                       rec=np.array([[8, 8, 8]], np.int32), precision=FP64)
        cp, cs = np.full((n, n, n), 3000.0, np.float32), np.full((n, n, n), 1700.0, np.float32)
        rho = np.empty((n, n, n), np.float32)
        rho[..., ::2], rho[..., 1::2] = r0, r1
        assert float(rho[0, 0, 0]) == r0 and float(rho[0, 0, 1]) == r1
        with Plan(p, cp, cs, rho, **tune) as plan:
            plan.run(2)
            before = plan.field(0, fp64=True)
            plan.run(1)
            after = plan.field(0, fp64=True)
            s = [plan.field(c, fp64=True) for c in (3, 6, 7)]
        b = float(2 * Fraction(dt) / (Fraction(r0) + Fraction(r1)))
        h = 1.0 / p.dx
        seen = 0
        for cell in np.ndindex(n - 8, n - 8, n - 8):
            cell = tuple(c + 4 for c in cell)
            if cell == (8, 8, 8):   # (the source adds to this one)
                continue
            want, t = rounded_vx(s, b, before[cell], h, h, h, cell)
            seen += t != 0.0
            assert after[cell] == want, (seed, cell, after[cell], want)
        assert seen > 20
