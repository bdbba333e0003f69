"""A plan with every tuning field open takes its tile and chunk from the grid
(plan_choice): results equal, bit for bit, the two half-step kernels on the
default tile, at grids where the rule changes sides -- each tile it can take,
widths and heights one off a tile's edge, claimed and dealt places, thin
grids, chunks down to two planes."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(p, cp, cs, rho, **kw):
    from ela3d_gb300 import Plan

    with Plan(p, cp, cs, rho, **kw) as plan:
        plan.run(7)
        plan.run(p.nstep - 7)
        return [plan.seismograms(), plan.source_trace()] + [plan.field(c) for c in range(9)]


@pytest.mark.parametrize("n", [
    (64, 64, 64),       # 64x14, two-plane chunks, dealt
    (80, 84, 33),       # 32x28
    (97, 29, 40),       # one column and one row past a 32x28 tile's edge
    (56, 33, 70),       # 56x16
    (113, 17, 50),      # one column past a 112-wide tile
    (127, 64, 90),      # 128x7
    (150, 211, 60),     # 32x28, claimed places
    (130, 150, 160),    # claimed, 64x14
    (3, 3, 3),
    (400, 5, 3),
])
@pytest.mark.parametrize("explosive", [False, True], ids=["force", "explosive"])
def test_open_plan_equals_two_kernels(n, explosive):
    from ela3d_gb300 import SRC_EXPLOSIVE, SRC_FORCE, STF_GAUSS_DERIV, STF_RICKER, ShotParams, media

    nx, ny, nz = n
    npml = max(0, min(8, (min(n) - 2) // 3))
    rng = np.random.default_rng(nx + ny + nz)
    rec = np.stack([rng.integers(0, m, 70) for m in n], axis=1).astype(np.int32)
    rec[:40, 2] = nz // 2   # many in the source's plane, some of them in its row
    rec[:12, 1] = ny // 3
    rec[0, 0] = nx // 2
    p = ShotParams(nx=nx, ny=ny, nz=nz, nstep=23, dt=1e-3, npml=npml, f0=25.0, t0=0.01, k_max=1.5,
                   src=(nx // 2, ny // 3, nz // 2), src_kind=SRC_EXPLOSIVE if explosive else SRC_FORCE,
                   stf=STF_GAUSS_DERIV if explosive else STF_RICKER, angle_force=25.0, rec=rec)
    cp, cs, rho = media.anticline_layers(nx, ny, nz, depths=(nz * 0.3, nz * 0.6, nz * 0.8, 2 * nz), amp=nz * 0.1,
                                         sigma=max(nx, ny) * 0.2, seed=3)
    want = _run(p, cp, cs, rho, variant=0, schedule=1, chunk=8)
    got = _run(p, cp, cs, rho)
    assert np.abs(want[0]).max() > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
