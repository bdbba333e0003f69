"""Page-locked model arrays wherever they lie in their locked range -- at its
start, up to its last byte, off a 16-byte boundary -- give the plans of ordinary
arrays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1], ids=["fp32", "fp64"])
@pytest.mark.parametrize("skip,tail", [(0, 0), (0, 5), (1, 0), (4, 0), (7, 3)])
@pytest.mark.parametrize("n", [(37, 20, 15), (32, 20, 15)], ids=["padded rows", "whole rows"])
def test_locked_model_equals_ordinary(built, n, skip, tail, precision):
    import ela3d_gb300 as E
    from ela3d_gb300 import media

    p = E.ShotParams(nx=n[0], ny=n[1], nz=n[2], nstep=25, dt=1e-3, npml=4, f0=25.0, t0=0.01, src=(18, 10, 7),
                     rec=np.array([[10, 10, 7], [25, 12, 9]], np.int32), precision=precision)
    m = media.anticline_layers(*n, depths=(4, 8, 12, 40), amp=2, sigma=8, seed=6)
    locked = []
    for a in m:
        whole = E.pinned_empty(skip + a.size + tail, np.float32)
        whole[:] = np.nan
        part = whole[skip:skip + a.size]
        part[:] = a.reshape(-1)
        assert part.ctypes.data == whole.ctypes.data + 4 * skip
        locked.append(part)
    got = []
    for model in (m, locked):
        with E.Plan(p, *model) as plan:
            plan.run(p.nstep)
            got.append([plan.seismograms()] + [plan.field(c) for c in range(9)])
    assert np.abs(got[0][0]).max() > 0
    for a, b in zip(*got):
        assert np.array_equal(a, b)
