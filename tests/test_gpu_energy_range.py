"""The energy of models and fields of any size FP32 holds: soft models, whose
moduli's products leave the range of doubles although every term of the sum is
ordinary, against the sum written out in numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def restated(p, cp, cs, rho, f):
    """Kinetic and strain energy cell by cell in float64, one division each."""
    cp, cs, rho = (a.astype(np.float64) for a in (cp, cs, rho))
    v, s = f[:3].astype(np.float64), f[3:].astype(np.float64)
    mu, lam = rho * cs * cs, rho * (cp * cp - 2.0 * cs * cs)
    ss = (s[:3] ** 2).sum(0) + 2.0 * (s[3:] ** 2).sum(0)
    tr = s[:3].sum(0)
    solid, fluid = mu > 0, (mu <= 0) & (lam > 0)
    m, l3 = np.where(solid, mu, 1.0), np.where(solid, 3.0 * lam + 2.0 * mu, 1.0)
    e = 0.5 * rho * (v ** 2).sum(0)
    e = e + np.where(solid, ss / (4.0 * m) - lam / (4.0 * m * l3) * tr * tr, 0.0)
    e = e + np.where(fluid, tr * tr / (18.0 * np.where(fluid, lam, 1.0)), 0.0)
    # (the plan holds 1 / dx in FP32)
    return e.sum() * np.prod([1.0 / float(np.float32(1) / np.float32(h)) for h in (p.dx, p.dy, p.dz)])


# (speeds and densities times these; the source times the last)
@pytest.mark.parametrize("speed,density,factor", [(1.0, 1.0, 1e7), (1e-25, 1.0, 1e7), (1e-26, 1.0, 1e7),
                                                  (1e-19, 1e-16, 1e3), (1e8, 1e11, 1e7)])
def test_energy_of_soft_and_hard_models(built, speed, density, factor):
    from ela3d_gb300 import Plan, ShotParams, media

    n = (21, 18, 16)   # (the last group of a row holds one cell)
    dt = 1e-3 / max(speed, 1.0)
    p = ShotParams(nx=n[0], ny=n[1], nz=n[2], nstep=12, dt=dt, npml=4, f0=0.05 / dt, t0=4 * dt, factor=factor,
                   src=(10, 9, 8), rec=np.array([[10, 9, 8]], np.int32))
    cp, cs, rho = media.anticline_layers(*n, depths=(5, 9, 13, 40), amp=2, sigma=6, seed=3)
    cs[0] = 0.0   # a fluid layer
    cp, cs, rho = (np.asarray(a * s, np.float32) for a, s in ((cp, speed), (cs, speed), (rho, density)))
    with Plan(p, cp, cs, rho) as plan:
        plan.run(p.nstep)
        got = plan.energy()
        f = np.stack([plan.field(c) for c in range(9)])
    want = restated(p, cp, cs, rho, f)
    assert np.isfinite(want) and want > 0
    assert abs(got - want) < 1e-12 * want
