"""The work lists of a running batch, which are built again whenever a shot
ends: a list whose allocation fails launches nothing, and the batch goes on from
there once there is memory again; time that passes with no shot left costs
nothing."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shots(precision=0):
    from ela3d_gb300 import ShotParams, media

    out = []
    for i, (n, steps) in enumerate([((40, 33, 30), 9), ((33, 40, 28), 31), ((48, 20, 25), 20)]):
        m = media.anticline_layers(*n, depths=(8, 15, 22, 60), amp=3, sigma=8, seed=i)
        out.append((ShotParams(nx=n[0], ny=n[1], nz=n[2], nstep=steps, dt=1e-3, npml=5, f0=25.0, t0=0.005,
                               src=(n[0] // 2, n[1] // 2, 12), rec=np.array([[n[0] // 3, n[1] // 2, 12]], np.int32),
                               precision=precision),) + tuple(m))
    return out


@pytest.mark.parametrize("precision", [0, 1], ids=["fp32", "fp64"])
@pytest.mark.parametrize("schedule", [-1, 1, 2, 4], ids=["open", "kind 1", "kind 2", "kind 4"])
@pytest.mark.parametrize("failures", [1, 2])
def test_failed_list_launches_nothing_and_the_batch_goes_on(built, schedule, precision, failures):
    from ela3d_gb300 import Batch, Ela3dError

    shots = _shots(precision)
    with Batch(shots, schedule=schedule) as b:
        b.run(31)
        want = [[b.seismograms(q), b.source_trace(q)] + [b.field(q, c) for c in range(9)] for q in range(3)]
    with Batch(shots, schedule=schedule) as b:
        b.run(10)   # (the first shot has ended: the dataflow kernel's list is built again now, the two kernels' at step 20)
        b.inject_list_failure(failures)
        for _ in range(failures):
            before = b.info(0).step
            with pytest.raises(Ela3dError) as e:
                b.run(31 - before)
            assert e.value.status == 2   # ELA3D_ERR_OOM
            assert before <= b.info(0).step < 31
        b.run(31 - b.info(0).step)
        got = [[b.seismograms(q), b.source_trace(q)] + [b.field(q, c) for c in range(9)] for q in range(3)]
    for g, w in zip(got, want):
        assert np.abs(w[0]).max() > 0
        for x, y in zip(g, w):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("schedule", [-1, 1], ids=["open", "two kernels"])
def test_time_passes_at_once_after_the_last_shot(built, schedule):
    from ela3d_gb300 import Batch

    shots = _shots()
    with Batch(shots, schedule=schedule) as b:
        b.run(31)
        done = [b.seismograms(q) for q in range(3)]
        t = time.perf_counter()
        b.run(1_000_000_000)
        assert time.perf_counter() - t < 5.0
        assert all(b.info(q).step == 1_000_000_031 for q in range(3))
        assert all(np.array_equal(b.seismograms(q), done[q]) for q in range(3))
        assert all(np.abs(d).max() > 0 for d in done)
