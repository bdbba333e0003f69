"""The choice of plans and batches whose tuning is left open
(ela3d_open_tuning): which tile a grid takes, and that each tile, taken that
way, gives the bits of the two half-step kernels."""
import numpy as np
import pytest

# a ragged grid for every tile the rule can take (FP32 and FP64, 152 SMs)
TILES = {
    (0, 128, 7): (118, 81, 73), (0, 128, 8): (118, 102, 58), (0, 112, 8): (105, 102, 65), (0, 112, 9): (99, 114, 62),
    (0, 64, 14): (169, 69, 60), (0, 64, 16): (182, 80, 48), (0, 56, 16): (163, 64, 67), (0, 56, 18): (151, 69, 67),
    (0, 32, 28): (94, 106, 70), (0, 32, 32): (87, 120, 67),
    (1, 8, 28): (81, 108, 80), (1, 16, 14): (106, 97, 68), (1, 16, 16): (126, 111, 50), (1, 32, 7): (87, 113, 71),
    (1, 32, 8): (127, 100, 55),
}
IDS = ["%s %dx%d" % ("fp64" if k[0] else "fp32", k[1], k[2]) for k in TILES]


def _params(n, **kw):
    import ela3d_gb300 as E

    rec = np.array([[n[0] // 2, n[1] // 3, n[2] // 2], [0, n[1] - 1, 0], [n[0] - 1, 0, n[2] - 1]], np.int32)
    return E.ShotParams(nx=n[0], ny=n[1], nz=n[2], nstep=23, dt=1e-3, npml=8, f0=25.0, t0=0.01, k_max=1.5,
                        src=(n[0] // 2, n[1] // 3, n[2] // 2), angle_force=25.0, rec=rec, **kw)


def _tile(t):
    import ela3d_gb300 as E

    v = E.variants()[t.variant]
    return v.tile_x, v.tile_y


@pytest.mark.parametrize("key", TILES, ids=IDS)
def test_each_grid_takes_its_tile(built, key):
    import ela3d_gb300 as E

    for kind in (E.SRC_FORCE, E.SRC_EXPLOSIVE):
        t = E.open_tuning(_params(TILES[key], precision=key[0], src_kind=kind))
        assert _tile(t) == key[1:] and t.schedule == 4 and t.chunk >= 2 and t.prefetch == 0
        assert E.variants()[t.variant].fp64 == key[0]


def test_named_sizes(built):
    """256^3 streams from HBM: both prefetches, chunks for two items per block;
    the FP64 cube takes the tile with the fewest idle threads."""
    import ela3d_gb300 as E
    from ela3d_gb300 import configs

    def pick(p):
        t = E.open_tuning(p)
        return _tile(t), t.schedule, t.chunk, t.prefetch

    assert pick(configs.anticline_256()[0]) == ((128, 8), 4, 52, 6)
    assert pick(configs.homogeneous_101()[0]) == ((112, 8), 4, 6, 0)   # 88% of the threads hold cells (112x9: 84%)
    assert pick(configs.homogeneous_101(precision=E.FP64)[0]) == ((8, 28), 4, 17, 0)
    assert pick(configs.anticline_256(n=128, precision=E.FP64)[0]) == ((16, 16), 4, 26, 0)


def test_prefetch_from_the_size_that_streams(built):
    """The line is 400 MB of arrays without the rows' padding: 201x201x206 lies
    below (399.5 MB; 445 with padding), one plane more above."""
    import ela3d_gb300 as E

    assert [E.open_tuning(_params((201, 201, nz))).prefetch for nz in (201, 206, 207)] == [0, 0, 6]


def test_batch_choice_up_to_the_most_shots_a_list_holds(built):
    """65535 shots share one dataflow list; more run on the two kernels."""
    import ela3d_gb300 as E

    p = E.ShotParams(nx=16, ny=16, nz=16, nstep=4, npml=2, src=(8, 8, 8))
    few = E.open_tuning(p, p)
    assert (few.schedule, few.chunk) == (4, 0)   # chunks are sized for the shots running
    shots = [p] * 65536
    assert E.open_tuning(*shots[1:]).schedule == 4
    many = E.open_tuning(*shots)
    assert (many.schedule, many.chunk) == (1, 10) and not E.variants()[many.variant].fp64


def test_open_tuning_rejects_what_creation_rejects(built):
    import ela3d_gb300 as E

    good = E.ShotParams(nx=16, ny=16, nz=16, nstep=4, npml=2, src=(8, 8, 8))
    for shots in ((good.with_(nx=2),), (good, good.with_(precision=1)), (good, good.with_(dt=-1.0)), ()):
        with pytest.raises(E.Ela3dError) as e:
            E.open_tuning(*shots)
        assert e.value.status == 1   # ELA3D_ERR_INVALID_ARG


@pytest.mark.gpu
@pytest.mark.parametrize("explosive", [False, True], ids=["force", "explosive"])
@pytest.mark.parametrize("key", TILES, ids=IDS)
def test_each_tile_taken_equals_two_kernels(built, key, explosive):
    """The open plan, and a plan created from ela3d_open_tuning's answer."""
    import ela3d_gb300 as E
    from ela3d_gb300 import media

    n, fp64 = TILES[key], key[0] == 1
    p = _params(n, precision=key[0], src_kind=E.SRC_EXPLOSIVE if explosive else E.SRC_FORCE)
    m = media.anticline_layers(*n, depths=(n[2] * 0.3, n[2] * 0.6, n[2] * 0.8, 2 * n[2]), amp=n[2] * 0.1,
                               sigma=max(n) * 0.2, seed=3)
    choice = E.open_tuning(p)
    assert _tile(choice) == key[1:]
    first = next(i for i, v in enumerate(E.variants()) if v.fp64 == key[0])
    out = []
    for tune in ({"variant": first, "schedule": 1, "chunk": 8}, {}, choice.as_dict()):
        with E.Plan(p, *m, **tune) as plan:
            plan.run(7)
            plan.run(p.nstep - 7)
            out.append([plan.seismograms(fp64=fp64), plan.source_trace(fp64=fp64)] +
                       [plan.field(c, fp64=fp64) for c in range(9)])
    assert np.abs(out[0][0]).max() > 0
    for got in out[1:]:
        for a, b in zip(got, out[0]):
            assert np.array_equal(a, b)
