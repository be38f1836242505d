"""Which kernels a system's steps take, by the launches it reports and counts, on both
sides of each size's line; and the pair-list step as one kernel on systems too large for
the cluster kernel, on batches, and beside steps with unequal radii.  (A system whose
displacement tracker has been started runs the two kernels, and so do profiled steps.)"""
import numpy as np
import pytest

from test_gpu_run_list import gas

pytestmark = pytest.mark.gpu


def system(psim, n, box, scale, precision=1, skin=0.3, vel_freq=25, rad=None, seed=5, up=True):
    g = psim.geometry(n, box, box / scale, scale)
    s = psim.System(g, psim.make_force("AO", 1.2, kT=1.0, well_depth=0.3), gamma=1.0, dt=0.001,
                    kT=1.0, vel_freq=vel_freq, seed=seed, precision=precision, skin=skin)
    if up:
        upload(s, n, box, rad)
    return s


def upload(s, n, box, rad=None):
    pos, r = gas(n, box, n)
    s.upload(pos, r if rad is None else rad,
             vel=np.random.default_rng(7).standard_normal(3 * n) * 2.0)


# the sizes of test_gpu_run_list.py and test_gpu_step_cells.py: kernels of a normal step,
# and of one with the tracker
@pytest.mark.parametrize("n,box,scale,precision,skin,normal,two", [
    (1, 9.0, 5, 1, 0.3, 1, 3), (8192, 34.0, 22, 1, 0.3, 1, 3), (8193, 34.0, 22, 1, 0.3, 2, 3),
    (700, 62.4, 38, 1, 0.3, 1, 3), (700, 65.6, 41, 1, 0.3, 2, 3),
    (1000, 18.0, 11, 0, 0.0, 2, 3), (16384, 45.0, 30, 0, 0.0, 2, 3), (16385, 45.0, 30, 0, 0.0, 3, 3),
    (24577, 50.0, 25, 0, 0.0, 7, 7), (24576, 50.0, 25, 1, 0.0, 2, 3), (24577, 50.0, 25, 1, 0.0, 6, 7),
    (393216, 126.0, 100, 1, 0.0, 6, 7), (393217, 126.0, 100, 1, 0.0, 7, 7)])
def test_kernels_of_a_step(psim, n, box, scale, precision, skin, normal, two):
    s = system(psim, n, box, scale, precision, skin)
    assert s.launches_per_step() == normal and s.launches_per_rebuild() == 0
    assert s.launches() == 0
    s.step(30)      # steps 0 and 26 are the first and a velocity step, as two kernels
    assert s.launches() == 2 * two + (
        1 + 3 * 2 if normal == 1 else 28 * normal)   # 25 in one launch, 3 are too few for one
    s.track_start()
    assert s.launches_per_step() == two
    s.close()


def test_kernels_with_lanes_and_unequal_radii(psim):
    n, box, scale = 1000, 18.0, 11
    s = system(psim, n, box, scale)
    s.set_list_lanes(2)
    assert s.launches_per_step() == 3
    s.set_list_lanes(1)
    assert s.launches_per_step() == 1
    upload(s, n, box, np.where(np.arange(n) % 2, 0.5, 0.45))
    assert s.launches_per_step() == 3
    s.close()


def outcome(s):
    return dict(s.download(), forces=s.forces(), at=np.array(s.get_step() + (s.list_builds(),)))


def same(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("n,box,scale", [(9000, 34.0, 22), (20001, 45.0, 30)])
@pytest.mark.parametrize("vel_freq", [3, 25, 1000])
def test_list_step_as_one_kernel(psim, n, box, scale, vel_freq):
    out = []
    for two in (False, True):
        s = system(psim, n, box, scale, vel_freq=vel_freq)
        if two:
            s.track_start()
        assert s.launches_per_step() == (3 if two else 2)
        for k in (1, 2, 17, 40, 5, 60, 1):
            s.step(k)
        out.append(outcome(s))
        s.close()
    same(*out)
    assert out[0]["at"][2] > 0


def test_batch_list_step_as_one_kernel(psim):
    sizes = [(9000, 34.0, 22), (300, 14.0, 9), (8193, 34.0, 22)]
    f = psim.make_force("AO", 1.2, kT=1.0, well_depth=0.3)
    parts = [gas(n, box, n) for n, box, _ in sizes]
    out = []
    for two in (False, True):
        b = psim.Batch([(psim.geometry(n, box, box / s, s), f, 5 + k)
                        for k, (n, box, s) in enumerate(sizes)], dt=0.001, kT=1.0, vel_freq=25,
                       skin=0.3)
        b.upload(np.concatenate([p for p, _ in parts]), np.concatenate([r for _, r in parts]),
                 vel=np.random.default_rng(7).standard_normal(3 * b.n) * 2.0)
        assert b.launches_per_step() == 2
        (b.profile if two else b.step)(126)
        out.append(outcome(b))
        b.close()
    same(*out)
    assert out[0]["at"][2] > 0


@pytest.mark.parametrize("n,box,scale", [(1000, 18.0, 11), (9000, 34.0, 22)])
def test_radii_change_with_an_upload(psim, n, box, scale):
    # equal radii (one kernel), unequal ones (two) and equal ones again on one system: the
    # bits of a system of its own each
    mixed = np.where(np.arange(n) % 2, 0.5, 0.45)
    s = system(psim, n, box, scale, up=False)
    for rad in (None, mixed, np.full(n, 0.48), None):
        upload(s, n, box, rad)
        s.step(60)
        one = system(psim, n, box, scale, rad=rad)
        one.step(60)
        same(outcome(s), outcome(one))
        one.close()
    s.close()
