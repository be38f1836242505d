"""The pair list's rebuild in the step's last kernel, at the edges of its blocks and of
its grid (608 blocks of 256 threads): after steps that rebuilt, the system's forces are
those of the FP64 pass on the oracle's own cells (the mixed form's tolerance), and a run
in single steps is the run in one call bit for bit."""
import numpy as np
import pytest

from gpu_helpers import FORCE_TOL_MIXED, rel_norm
from oracle import port
from test_gpu_run_list import gas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box,scale", [(255, 14.0, 9), (257, 14.0, 9), (8193, 34.0, 22),
                                         (20001, 46.0, 30), (155648, 92.0, 61), (155649, 92.0, 3),
                                         (20001, 90.0, 60)])
def test_forces_after_rebuilds(psim, n, box, scale):
    pos, rad = gas(n, box, n)
    vel = np.random.default_rng(7).standard_normal(3 * n) * 2.0
    p = psim.make_force("AO", 1.2, kT=1.0, well_depth=0.3)
    g = psim.geometry(n, box, box / scale, scale)
    out = []
    for steps in ((60,), (1,) * 60):
        s = psim.System(g, p, gamma=1.0, dt=0.001, kT=1.0, vel_freq=25, seed=5, skin=0.3)
        s.upload(pos, rad, vel=vel)
        s.track_start()   # a small system too runs this kernel
        for k in steps:
            s.step(k)
        assert s.list_builds() > 0
        out.append((s.download()["pos"], s.forces()))
        s.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    x, f = out[0]
    og = port.geom(n, box, box / scale, scale)
    hi, cse, srt = port.build_cells(og, x, rad)
    assert rel_norm(f, psim.force_evaluate(p, g, srt, hi, cse)) <= FORCE_TOL_MIXED
