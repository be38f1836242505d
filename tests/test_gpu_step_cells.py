"""The step without a pair list as one kernel (small systems) against the force pass and
the update as two: the same bits, at the edges of a warp's eight particles and of the
sizes it takes, with velocity steps and with injected noise.  (A system whose displacement
tracker has been started runs the two kernels.)"""
import numpy as np
import pytest

from test_gpu_run_list import gas

pytestmark = pytest.mark.gpu

KINDS = {"AO": lambda psim: psim.make_force("AO", 1.2, kT=1.0, well_depth=0.3),
         "LJ6": lambda psim: psim.make_force("LJ", 1.2, kT=1.0, well_depth=0.5, lj_num=6,
                                             yukawa_strength=0.0),
         "LJ9Y": lambda psim: psim.make_force("LJ", 1.5, kT=1.0, well_depth=0.5, lj_num=9,
                                              yukawa_strength=1.0),
         "CAL": lambda psim: psim.make_force("CAL", 1.1),
         "AO_YUK": lambda psim: psim.make_force("AO_YUK", 1.1, well_depth=0.2, cutoff2=1.5,
                                                well_depth2=1.0, yukawa_strength=5.0,
                                                debye_length=0.3, lj_num=0)}


def both(psim, n, box, scale, kind, vel_freq, noise=None, precision="FP64"):
    pos, rad = gas(n, box, n)
    vel = np.random.default_rng(7).standard_normal(3 * n) * 2.0
    g = psim.geometry(n, box, box / scale, scale)
    out = []
    for two in (False, True):
        s = psim.System(g, KINDS[kind](psim), gamma=1.0, dt=0.001, kT=1.0, vel_freq=vel_freq,
                        seed=5, precision=getattr(psim, "PRECISION_" + precision), skin=0.0,
                        noise_mode=0 if noise is None else psim.NOISE_INJECTED)
        s.upload(pos, rad, vel=vel)
        if noise is not None:
            s.set_noise(noise, len(noise))
        if two:
            s.track_start()
        try:
            for k in (1, 2, 17, 40, 5):
                s.step(k)
        except psim.PsimError as e:
            out.append((e.code, str(e), s.get_step()))
        else:
            out.append((s.download(), s.forces(), s.get_step()))
        s.close()
    (a, fa, ta), (b, fb, tb) = out
    assert ta == tb
    if isinstance(a, int):
        assert (a, fa) == (b, fb)
        return a, ta
    for k in ("pos", "pos0", "vel", "frc", "frc0"):
        assert np.array_equal(a[k], b[k]), k
    assert np.array_equal(fa, fb)
    return 0, ta


@pytest.mark.parametrize("n,box,scale", [(1, 9.0, 5), (7, 9.0, 5), (17, 9.0, 5), (513, 14.0, 9),
                                         (4097, 28.0, 18), (16384, 45.0, 30), (16385, 45.0, 30),
                                         (24577, 50.0, 30), (393216, 126.0, 100),
                                         (393217, 126.0, 100)])
@pytest.mark.parametrize("vel_freq", [0, 4, 25])
@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_one_kernel_steps_as_two(psim, n, box, scale, vel_freq, precision):
    code, at = both(psim, n, box, scale, "AO", vel_freq, precision=precision)
    assert code == 0 and at[0] == 65


@pytest.mark.parametrize("kind", ["LJ6", "LJ9Y", "CAL", "AO_YUK"])
@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_plugins(psim, kind, precision):
    both(psim, 1000, 18.0, 11, kind, 25, precision=precision)


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_injected_noise_ends(psim, precision):
    noise = np.random.default_rng(3).standard_normal((40, 6 * 300))
    code, at = both(psim, 300, 14.0, 9, "AO", 1000, noise=noise, precision=precision)
    assert code == psim.ERR_INPUT and at[0] == 40
