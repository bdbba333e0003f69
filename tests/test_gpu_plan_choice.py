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
    (130, 150, 160),    # claimed, 64-wide
    (128, 32, 60),      # 128x8, eight consumer warps
    (192, 48, 40),      # 64x16
    (160, 64, 40),      # 32x32
    (201, 63, 33),      # 112x9, whose last threads have no cells
    (112, 36, 40),      # 56x18 or 112x9, one row past a tile's edge less
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


@pytest.mark.parametrize("n", [(32, 14, 20), (33, 15, 64), (16, 28, 70), (101, 101, 33), (9, 57, 40), (3, 3, 3), (32, 16, 40),
                               (64, 8, 33)])
@pytest.mark.parametrize("explosive", [False, True], ids=["force", "explosive"])
def test_open_fp64_plan_equals_two_kernels(n, explosive):
    """The same in FP64: each of its tiles and one cell past their edges."""
    import ela3d_gb300 as E
    from ela3d_gb300 import media

    nx, ny, nz = n
    p = E.ShotParams(nx=nx, ny=ny, nz=nz, nstep=23, dt=1e-3, npml=max(0, min(8, (min(n) - 2) // 3)), f0=25.0, t0=0.01,
                     k_max=1.5, src=(nx // 2, ny // 3, nz // 2), precision=E.FP64, angle_force=25.0,
                     src_kind=E.SRC_EXPLOSIVE if explosive else E.SRC_FORCE,
                     rec=np.array([[nx // 2, ny // 3, nz // 2], [0, ny - 1, 0], [nx - 1, 0, nz - 1]], np.int32))
    cp, cs, rho = media.anticline_layers(nx, ny, nz, depths=(nz * 0.3, nz * 0.6, nz * 0.8, 2 * nz), amp=nz * 0.1,
                                         sigma=max(nx, ny) * 0.2, seed=3)
    first = next(i for i, v in enumerate(E.variants()) if v.fp64)
    want = _run(p, cp, cs, rho, variant=first, schedule=1, chunk=8)
    got = _run(p, cp, cs, rho)
    assert np.abs(want[0]).max() > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_open_batch_equals_shots_alone(built):
    """A batch with open tuning: uneven grids, lengths and source kinds (the
    shots that end first are passed over), and two shots of one model."""
    import ela3d_gb300 as E
    from ela3d_gb300 import media

    shots = []
    for i, (n, steps, kind) in enumerate([((70, 33, 90), 31, 0), ((33, 64, 40), 9, 1), ((129, 15, 60), 57, 0),
                                          ((70, 33, 90), 44, 0)]):
        m = shots[0][1:] if i == 3 else media.anticline_layers(
            *n, depths=(n[2] * 0.3, n[2] * 0.7, n[2], 2 * n[2]), amp=4, sigma=n[0] * 0.2, seed=i)
        rec = np.array([[n[0] // 2, n[1] // 2, 12 + q] for q in range(5)], np.int32)
        shots.append((E.ShotParams(nx=n[0], ny=n[1], nz=n[2], nstep=steps, dt=1e-3, npml=5, f0=25.0, t0=0.005,
                                   src=(n[0] // 2, n[1] // 2, 12), src_kind=kind, rec=rec), *m))
    for group in (shots, [s for s in shots if s[0].src_kind == E.SRC_FORCE]):
        with E.Batch(group) as b:
            b.run(20)
            b.run(40)
            for q, s in enumerate(group):
                with E.Plan(*s, variant=0, schedule=1, chunk=8) as plan:
                    plan.run(s[0].nstep)
                    assert np.array_equal(b.seismograms(q), plan.seismograms())
                    assert np.array_equal(b.source_trace(q), plan.source_trace())
                    for c in range(9):
                        assert np.array_equal(b.field(q, c), plan.field(c)), (q, c)


@pytest.mark.parametrize("scale", [1e-36, 1e-20, 1.0, 1e30])
def test_fp64_densities_of_any_size(built, scale):
    """The FP64 kernels' own dt / rho quotient and, for sums of densities
    outside its range (1e-36 and 1e30 kg/m^3 times the usual), the general
    division, against the FP64 oracle: the tolerance of the FP64 parity tests."""
    import oracle
    from conftest import rel_l2
    from ela3d_gb300 import FP64, Plan, ShotParams, media

    nx, ny, nz = 37, 30, 33
    p = ShotParams(nx=nx, ny=ny, nz=nz, nstep=40, dt=1e-3, npml=6, f0=25.0, t0=0.02, src=(18, 15, 16),
                   rec=np.array([[10, 15, 16], [25, 20, 10]], np.int32), precision=FP64)
    cp, cs, rho = media.anticline_layers(nx, ny, nz, depths=(8, 15, 24, 60), amp=3, sigma=8, seed=4)
    rho = (rho.astype(np.float64) * scale).astype(np.float32)
    want, fields = oracle.run(p, cp, cs, rho, p.nstep, fp64=True)
    with Plan(p, cp, cs, rho) as plan:
        plan.run(p.nstep)
        assert np.abs(want).max() > 0 and rel_l2(plan.seismograms(fp64=True), want) < 1e-11
        for c in range(9):
            assert rel_l2(plan.field(c, fp64=True), fields[c]) < 1e-11, c


def test_fp64_coefficients_follow_a_restored_model(built):
    """An FP64 plan on the dataflow kernel runs from coefficients derived from
    its model; a checkpoint brings its own model, and the plan then continues
    as the saved one.  A batch's shots of one model share them, also when their
    time steps differ."""
    import ela3d_gb300 as E
    from ela3d_gb300 import media

    nx, ny, nz = 48, 40, 36
    p = E.ShotParams(nx=nx, ny=ny, nz=nz, nstep=30, dt=1e-3, npml=6, f0=25.0, t0=0.01, src=(24, 20, 18),
                     rec=np.array([[20, 20, 18], [30, 22, 12]], np.int32), precision=E.FP64)
    m = media.anticline_layers(nx, ny, nz, depths=(10, 20, 30, 60), amp=3, sigma=9, seed=1)
    other = media.anticline_layers(nx, ny, nz, depths=(8, 15, 22, 60), amp=4, sigma=7, seed=2)
    first = next(i for i, v in enumerate(E.variants()) if v.fp64)
    want = _run(p, *m, variant=first, schedule=1, chunk=8)
    with E.Plan(p, *m) as a:
        a.run(12)
        saved = a.checkpoint()
    with E.Plan(p, *other) as b:
        b.restore(saved)
        b.run(p.nstep - 12)
        got = [b.seismograms(), b.source_trace()] + [b.field(c) for c in range(9)]
    for x, y in zip(got, want):
        assert np.array_equal(x, y)
    shots = [(p, *m), (p.with_(dt=0.8e-3, src=(20, 18, 16)), *m), (p.with_(src=(30, 20, 16)), *m)]
    with E.Batch(shots) as b:
        b.run(p.nstep)
        for q, s in enumerate(shots):
            alone = _run(*s, variant=first, schedule=1, chunk=8)
            assert np.array_equal(b.seismograms(q), alone[0])
            assert np.array_equal(b.field(q, 2), alone[4])


@pytest.mark.parametrize("nz", [133, 134], ids=["hinted", "plain"])
@pytest.mark.parametrize("tile", [(128, 7), (64, 14), (112, 8), (56, 16), (32, 28), (128, 8), (64, 16), (32, 32),
                                  (112, 9), (56, 18)], ids=lambda t: "%dx%d" % t)
def test_l2_hints_equal_two_kernels(tile, nz):
    """128x128xnz: the arrays of 133 planes are just below the size up to which
    the dataflow kernel runs with L2 hints, those of 134 just above."""
    from ela3d_gb300 import ShotParams, media, variants

    rec = np.stack([np.arange(40, 80), np.full(40, 60), np.full(40, 66)], axis=1).astype(np.int32)
    p = ShotParams(nx=128, ny=128, nz=nz, nstep=9, dt=1e-3, npml=12, f0=25.0, t0=0.004, k_max=1.5, src=(63, 60, 66),
                   rec=rec)
    cp, cs, rho = media.anticline_layers(128, 128, nz, depths=(40, 80, 100, 2 * nz), amp=13, sigma=26, seed=4)
    number = next(i for i, v in enumerate(variants()) if (v.tile_x, v.tile_y) == tile and not v.fp64 and v.loads == 0)
    want = _run(p, cp, cs, rho, variant=0, schedule=1, chunk=8)
    got = _run(p, cp, cs, rho, variant=number, schedule=4, chunk=12)
    assert np.abs(want[0]).max() > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
