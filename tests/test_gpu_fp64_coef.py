"""FP64 tiles on the dataflow kernel, with update coefficients from arrays and
with the kernel's own (ELA3D_COEF_BYTES=0, what a plan runs that finds no room
for the arrays), and a batch of which only the first shot has them: the bits of
the two half-step kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILES = [(32, 7), (32, 3), (32, 6), (64, 3), (16, 14), (8, 28), (32, 8), (16, 16)]


def _variant(tile):
    import ela3d_gb300 as E

    return next(i for i, v in enumerate(E.variants()) if v.fp64 and (v.tile_x, v.tile_y) == tile)


def _shot(n, explosive=False, seed=3, **kw):
    import ela3d_gb300 as E
    from ela3d_gb300 import media

    p = E.ShotParams(nx=n[0], ny=n[1], nz=n[2], nstep=17, dt=1e-3, npml=max(0, min(5, (min(n) - 2) // 3)), f0=25.0,
                     t0=0.006, k_max=1.5, src=(n[0] // 2, n[1] // 3, n[2] // 2), precision=E.FP64, angle_force=25.0,
                     src_kind=E.SRC_EXPLOSIVE if explosive else E.SRC_FORCE,
                     rec=np.array([[n[0] // 2, n[1] // 3, n[2] // 2], [0, n[1] - 1, 0], [n[0] - 1, 0, n[2] - 1]], np.int32),
                     **kw)
    m = media.anticline_layers(*n, depths=(n[2] * 0.3, n[2] * 0.6, n[2] * 0.8, 2 * n[2]), amp=n[2] * 0.1,
                               sigma=max(n) * 0.2, seed=seed)
    return (p,) + tuple(m)


def _results(p, *m, **tune):
    from ela3d_gb300 import Plan

    with Plan(p, *m, **tune) as plan:
        plan.run(6)
        plan.run(p.nstep - 6)
        return plan.info().device_bytes, [plan.seismograms(fp64=True), plan.source_trace(fp64=True)] + [
            plan.field(c, fp64=True) for c in range(9)]


def _coef_bytes(p):
    return 64 * -(-p.nx // 16) * 16 * p.ny * p.nz


@pytest.mark.parametrize("explosive", [False, True], ids=["force", "explosive"])
@pytest.mark.parametrize("size", ["below", "at", "above"])
@pytest.mark.parametrize("tile", TILES, ids=lambda t: "%dx%d" % t)
def test_tile_with_and_without_coefficients(built, monkeypatch, tile, size, explosive):
    tx, ty = tile
    n = {"below": (2 * tx - 1, 2 * ty - 1, 19), "at": (tx, 2 * ty, 20), "above": (2 * tx + 1, ty + 1, 21)}[size]
    shot = _shot(n, explosive)
    bytes0, want = _results(*shot, variant=_variant((32, 7)), schedule=1, chunk=8)
    # (tiles of two cells a thread, and the one of two blocks per SM, are not compiled with arrays)
    arrays = tile not in ((32, 6), (64, 3), (32, 3))
    assert np.abs(want[0]).max() > 0
    for budget in (None, "0"):
        if budget is not None:
            monkeypatch.setenv("ELA3D_COEF_BYTES", budget)
        held, got = _results(*shot, variant=_variant(tile), schedule=4, chunk=4)
        assert held - bytes0 == (_coef_bytes(shot[0]) if budget is None and arrays else 0)
        for a, b in zip(got, want):
            assert np.array_equal(a, b), budget


def test_batch_of_which_one_shot_has_coefficients(built, monkeypatch):
    import ela3d_gb300 as E

    shots = [_shot((40, 30, 24)), _shot((40, 30, 24), seed=4), _shot((33, 18, 20), explosive=True)]
    monkeypatch.setenv("ELA3D_COEF_BYTES", str(_coef_bytes(shots[0][0])))
    with E.Batch(shots) as b:
        b.run(17)
        got = [[b.seismograms(q)] + [b.field(q, c) for c in range(9)] for q in range(3)]
        held = [b.info(q).device_bytes for q in range(3)]
    for q, s in enumerate(shots):
        with E.Plan(*s, variant=_variant((32, 7)), schedule=1, chunk=8) as plan:
            plan.run(17)
            want = [plan.seismograms()] + [plan.field(c) for c in range(9)]
            assert held[q] - plan.info().device_bytes == (_coef_bytes(s[0]) if q == 0 else 0)
        assert np.abs(want[0]).max() > 0
        for a, w in zip(got[q], want):
            assert np.array_equal(a, w), q


@pytest.mark.parametrize("precision,tile", [(0, t) for t in ((128, 8), (64, 16), (32, 32), (112, 9), (56, 18), (32, 28))] +
                         [(1, t) for t in ((16, 16), (32, 8), (8, 28), (16, 14))])
def test_nan_padding_never_reaches_the_grid(built, precision, tile):
    """The tiles of eight warps, and FP64 from coefficients, with NaN in every
    padding column of the fields and memory variables."""
    import ela3d_gb300 as E

    n = (37, 33, 18)
    p, *m = _shot(n)
    p = p.with_(precision=precision)
    variant = next(i for i, v in enumerate(E.variants())
                   if v.fp64 == precision and not v.loads and (v.tile_x, v.tile_y) == tile)
    for schedule in (1, 4):
        out = []
        for poison in (False, True):
            with E.Plan(p, *m, variant=variant, schedule=schedule, chunk=4) as plan:
                if poison:
                    plan.poison_padding(float("nan"))
                plan.run(p.nstep)
                out.append([plan.seismograms(fp64=precision == 1)] +
                           [plan.field(c, fp64=precision == 1) for c in range(9)])
        for a, b in zip(*out):
            assert np.all(np.isfinite(b)) and np.array_equal(a, b)
