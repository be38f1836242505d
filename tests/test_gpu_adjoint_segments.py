"""The adjoint's stored trajectory: a run too long to be kept whole (three segments, the
first two recomputed) against the same run kept whole at the caller's wish."""
import math

import numpy as np
import pytest

from test_gpu_adjoint import _lj_params

pytestmark = pytest.mark.gpu


def test_segments_as_the_whole_trajectory(psim):
    from proteinsim2015_gb300 import adjoint as adj
    from proteinsim2015_gb300 import init
    n, T = 32768, 400      # 256 MB hold 170 steps
    box = (n * math.pi / 6.0 / 0.15) ** (1.0 / 3.0)
    scale = int(box // 3.1)
    g = psim.geometry(n, box, box / scale, scale)
    pos = init.rsa_native(n, box, 1.0, seed=n).reshape(-1)
    vel = init.maxwell(n, 1.0, seed=n).reshape(-1)
    p, _ = _lj_params(adj)
    out = []
    for K in (50, T):
        a = adj.Adjoint(g, T, dt=0.001, seed=3, checkpoint_every=K, sample_every=50)
        out.append(a.gradient(p, pos, np.ones(100), vel, wrt_pos=True))
        out[-1] += (a.forward(p, pos, vel),)
        a.close()
    (la, ga, da, xa, fa), (lb, gb, db, xb, fb) = out
    # the same arithmetic on lists built at other steps: rounding, and its growth over
    # the trajectory
    assert la == pytest.approx(lb, rel=1e-9)
    assert np.allclose(ga, gb, rtol=1e-9, atol=1e-12)
    assert np.allclose(fa, ga, rtol=1e-9, atol=1e-12) and np.allclose(fb, gb, rtol=1e-9, atol=1e-12)
    assert np.allclose(da, db, rtol=1e-6, atol=1e-9 * np.max(np.abs(db)))
    assert np.linalg.norm(xa - xb) <= 1e-6 * np.linalg.norm(xb)
