"""The pair-list step as one kernel against the force pass and the update as two:
the same bits, through list rebuilds, velocity steps and runs that begin and end
anywhere in a buffer period.  (A system whose displacement tracker has been
started runs the two kernels.)"""
import numpy as np
import pytest

from gpu_helpers import lattice_state, rsa_state

pytestmark = pytest.mark.gpu


def state_of(kind, n):
    if kind == "LJ":
        pos, rad, box = lattice_state(9, (4 / 0.8) ** (1 / 3), 0.1, seed=n)
        keep = np.sort(np.random.default_rng(n).permutation(len(rad))[:n])
        return pos.reshape(-1, 3)[keep].reshape(-1), rad[:n], box
    pos, rad = rsa_state(n, 14.0, seed=n)
    return pos, rad, 14.0


def force_of(psim, kind):
    if kind == "LJ":
        return psim.make_force("LJ", 2.5, kT=1.5, well_depth=1 / 1.5, lj_num=6, yukawa_strength=0.0)
    if kind == "LJY":
        return psim.make_force("LJ", 2.5, kT=1.0, well_depth=2.0, lj_num=7, yukawa_strength=3.0)
    return psim.make_force("AO", 1.2, kT=1.0, well_depth=0.3)


@pytest.mark.parametrize("kind,n", [("AO", 1), ("AO", 255), ("LJY", 257), ("LJ", 2916), ("AO", 1000)])
@pytest.mark.parametrize("vel_freq", [0, 4, 25])
def test_one_kernel_steps_as_two(psim, kind, n, vel_freq):
    pos, rad, box = state_of(kind, n)
    p = force_of(psim, kind)
    scale = int(box / (p.cutoff + 0.3))
    g = psim.geometry(n, box, box / scale, scale)
    vel = np.random.default_rng(7).standard_normal(3 * n) * 3.0   # rebuilds within a few steps
    out = []
    for two in (False, True):
        s = psim.System(g, p, gamma=1.0, dt=0.001, kT=1.0, vel_freq=vel_freq, seed=5, skin=0.3)
        s.upload(pos, rad, vel=vel)
        if two:
            s.track_start()
        try:
            for k in (1, 2, 17, 40, 5, 60, 1):
                s.step(k)
        except psim.PsimError as e:   # the fast liquid may run into an overlap: the same one
            out.append((e.code, str(e), s.list_builds(), s.get_step()))
        else:
            out.append((s.download(), s.forces(), s.list_builds(), s.get_step()))
        s.close()
    (a, fa, la, ta), (b, fb, lb, tb) = out
    assert la == lb and ta == tb
    assert n < 200 or la > 0
    if isinstance(a, int):
        assert (a, fa) == (b, fb) and kind == "LJ" and ta[0] > 0
        return
    for k in ("pos", "pos0", "vel", "frc", "frc0"):
        assert np.array_equal(a[k], b[k]), k
    assert np.array_equal(fa, fb)


def test_overlap_leaves_the_state_of_the_failing_step(psim):
    # two particles shot at each other among bystanders: the step that finds them
    # closer than 0.8 diameters reports it, and the state is that step's start
    n, box, scale = 300, 14.0, 9
    pos, rad = rsa_state(n, box, seed=3)
    pos[:6] = [1.0, 7.0, 7.0, 2.3, 7.0, 7.0]
    d = pos.reshape(-1, 3)[2:, None] - pos.reshape(-1, 3)[None, :2]
    d -= box * np.round(d / box)
    keep = np.concatenate([[True, True], np.all(np.linalg.norm(d, axis=2) > 1.6, axis=1)])
    pos, n = pos.reshape(-1, 3)[keep].reshape(-1), int(keep.sum())
    vel = np.zeros(3 * n)
    vel[0], vel[3] = 120.0, -120.0
    p = psim.make_force("CAL", 1.1)
    g = psim.geometry(n, box, box / scale, scale)
    out = []
    for two in (False, True):
        s = psim.System(g, p, gamma=1.0, dt=0.001, kT=1.0, vel_freq=1000, seed=5, skin=0.3)
        s.upload(pos, np.full(n, 0.5), vel=vel)
        if two:
            s.track_start()
        with pytest.raises(psim.PsimError) as e:
            s.step(40)
        assert e.value.code == psim.ERR_OVERLAP
        step = s.get_step()
        try:
            st = s.download()
        except psim.PsimError:
            st = None
        out.append((step, st))
        s.close()
    assert out[0][0] == out[1][0]
    if out[0][1] is not None:
        for k in ("pos", "pos0", "vel"):
            assert np.array_equal(out[0][1][k], out[1][1][k]), k
