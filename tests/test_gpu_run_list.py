"""Stretches of normal steps of a small system in one kernel against the force pass and
the update as two kernels a step: the same bits, at the edges of the sizes it takes, in
every schedule, with injected noise and through list rebuilds.  (A system whose
displacement tracker has been started runs the two kernels.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def gas(n, box, seed):
    m = int(np.ceil(n ** (1 / 3)))
    i = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(seed)
    i = i[np.sort(rng.permutation(len(i))[:n])]
    a = box / m
    return np.mod((i + 0.5) * a + rng.uniform(-0.1, 0.1, (n, 3)), box).reshape(-1), np.full(n, 0.5)


def both(psim, n, box, scale, force, steps, vel_freq, noise=None):
    pos, rad = gas(n, box, n)
    vel = np.random.default_rng(7).standard_normal(3 * n) * 2.0
    g = psim.geometry(n, box, box / scale, scale)
    out = []
    for two in (False, True):
        s = psim.System(g, force, gamma=1.0, dt=0.001, kT=1.0, vel_freq=vel_freq, seed=5,
                        skin=0.3, noise_mode=0 if noise is None else psim.NOISE_INJECTED)
        s.upload(pos, rad, vel=vel)
        if noise is not None:
            s.set_noise(noise, len(noise))
        if two:
            s.track_start()
        try:
            for k in steps:
                s.step(k)
        except psim.PsimError as e:
            out.append((e.code, str(e), s.list_builds(), s.get_step()))
        else:
            out.append((s.download(), s.forces(), s.list_builds(), s.get_step()))
        s.close()
    (a, fa, la, ta), (b, fb, lb, tb) = out
    assert la == lb and ta == tb
    if isinstance(a, int):
        assert (a, fa) == (b, fb)
        return a, ta
    for k in ("pos", "pos0", "vel", "frc", "frc0"):
        assert np.array_equal(a[k], b[k]), k
    assert np.array_equal(fa, fb)
    return la, ta


# one particle; one warp a block and one more; the most it takes and one more; the
# most cells it takes with 700 particles and more (38^3, 39^3); three cells a side
@pytest.mark.parametrize("n,box,scale", [(1, 9.0, 5), (33, 9.0, 5), (512, 14.0, 9), (513, 14.0, 9),
                                         (4097, 28.0, 18), (8192, 34.0, 22), (8193, 34.0, 22),
                                         (700, 64.0, 40), (700, 65.6, 41), (700, 60.8, 38),
                                         (700, 62.4, 39), (64, 7.0, 3)])
@pytest.mark.parametrize("vel_freq", [1, 25, 1000])
def test_same_bits(psim, n, box, scale, vel_freq):
    builds, at = both(psim, n, box, scale, psim.make_force("AO", 1.2, kT=1.0, well_depth=0.3),
                  (1, 2, 17, 40, 5, 60, 1), vel_freq)
    assert at[0] == 126 and (n < 500 or builds > 0)


@pytest.mark.parametrize("kind", ["LJ6", "LJ9Y", "CAL"])
def test_plugins(psim, kind):
    force = {"LJ6": lambda: psim.make_force("LJ", 1.2, kT=1.0, well_depth=0.5, lj_num=6,
                                            yukawa_strength=0.0),
             "LJ9Y": lambda: psim.make_force("LJ", 1.2, kT=1.0, well_depth=0.5, lj_num=9,
                                             yukawa_strength=1.0),
             "CAL": lambda: psim.make_force("CAL", 1.1)}[kind]()
    assert both(psim, 1000, 18.0, 12, force, (100, 30), 25)[0] > 0


def test_more_steps_than_one_launch_takes(psim):
    assert both(psim, 300, 14.0, 9, psim.make_force("AO", 1.2, kT=1.0, well_depth=0.3), (2500,),
                100000)[0] > 0


def test_injected_noise(psim):
    # steps 0..39 have noise; the one after them reports that it has none, and the
    # state stays where it was
    noise = np.random.default_rng(3).standard_normal((40, 6 * 300))
    ao = psim.make_force("AO", 1.2, kT=1.0, well_depth=0.3)
    both(psim, 300, 14.0, 9, ao, (40,), 25, noise=noise)
    code, at = both(psim, 300, 14.0, 9, ao, (60,), 1000, noise=noise)
    assert code == psim.ERR_INPUT and at[0] == 40
