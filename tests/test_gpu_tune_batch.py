"""Tuning a batch never leaves later batches of its shape on a choice that was
measured slower than the open one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import ela3d_gb300 as E
from ela3d_gb300 import configs

shots, cp, cs, rho = configs.anticline_256_shots(3, nstep=40, n=64)
shots = [(s, cp, cs, rho) for s in shots]
if sys.argv[3] == "call":
    best, ms, cand = E.autotune(shots, steps=20)
    assert best.schedule in (0, 1, 2) and ms > 0
tune = {"schedule": 1} if sys.argv[3] == "partly" else {}
with E.Batch(shots, **tune) as b:
    b.run(40)
    np.save(sys.argv[2], np.stack([b.field(q, c) for q in range(3) for c in range(9)]))
"""


def test_cache_holds_the_faster_open_choice(built, tmp_path):
    """Three 64^3 shots, where the dataflow kernel is far ahead of two launches
    a step: the cache gets the open choice (schedule 4, chunk 0), from an
    autotuner call and from ELA3D_AUTOTUNE=1, and a fresh process runs on it;
    one that sets a field does not take its chunk."""
    import os
    import subprocess
    import sys

    import ela3d_gb300 as E
    from ela3d_gb300 import configs

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    prog = tmp_path / "child.py"
    prog.write_text(CHILD)
    shots = configs.anticline_256_shots(3, nstep=40, n=64)[0]
    choice = E.open_tuning(*shots)
    out = {}
    for how in ("open", "call", "cached", "env", "partly"):
        cache = tmp_path / ("env.txt" if how in ("env", "partly") else "call.txt")
        env = dict(os.environ)
        env.pop("ELA3D_AUTOTUNE", None)
        env.pop("ELA3D_TUNE_CACHE", None)
        if how != "open":
            env["ELA3D_TUNE_CACHE"] = str(cache)
        if how == "env":
            env["ELA3D_AUTOTUNE"] = "1"
        r = subprocess.run([sys.executable, str(prog), root, str(tmp_path / (how + ".npy")), how], env=env,
                           capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        out[how] = np.load(tmp_path / (how + ".npy"))
        if how != "open":
            key, *entry = cache.read_text().split()
            assert key.startswith("0:3:64x64x64") and [int(v) for v in entry] == [choice.variant, 4, 0, 0, 0, 0]
    assert np.abs(out["open"]).max() > 0
    for how in out:
        assert np.array_equal(out[how], out["open"]), how
