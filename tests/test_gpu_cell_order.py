"""The cell order of a system without a pair list, made by one kernel up to its limits
and by several beyond: after a few steps the system's forces are, bit for bit, those of
the force pass on the oracle's sorted particles (cells in order, tags within a cell)."""
import numpy as np
import pytest

from gpu_helpers import oracle_force
from oracle import port

pytestmark = pytest.mark.gpu

ORDER_MAX = 3 << 13


# one particle; a block's slice and one more; several rounds of a block's threads; the
# most cells it takes with 700 particles and more (38^3, 39^3); the most particles and more
@pytest.mark.parametrize("n,box,scale", [(1, 9.0, 5), (511, 9.0, 5), (513, 9.0, 5), (4097, 28.0, 18),
                                         (16385, 45.0, 30), (700, 60.8, 38), (700, 62.4, 39),
                                         (700, 64.0, 40), (700, 65.6, 41), (65535, 66.0, 40),
                                         (65537, 66.0, 40), (ORDER_MAX, 45.0, 29),
                                         (ORDER_MAX + 1, 45.0, 29)])
def test_canonical_order(psim, n, box, scale):
    m = int(np.ceil(n ** (1 / 3)))
    i = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(n)
    i = rng.permutation(i)[:n]   # tags in no spatial order
    pos = np.mod((i + 0.5) * (box / m) + rng.uniform(-0.1, 0.1, (n, 3)), box).reshape(-1)
    rad = np.full(n, 0.45)
    p = psim.make_force("AO", 1.2, kT=1.0, well_depth=0.3)
    g = psim.geometry(n, box, box / scale, scale)
    s = psim.System(g, p, gamma=1.0, dt=0.001, kT=1.0, seed=5, precision=psim.PRECISION_FP64, skin=0.0)
    s.upload(pos, rad, vel=rng.standard_normal(3 * n) * 20.0)   # cells change within a step
    for k in (1, 2, 4):
        try:
            s.step(k)
        except psim.PsimError as e:   # the crowded ones run into an overlap after a few steps
            assert e.code == psim.ERR_OVERLAP and k == 4
            break
        x = s.download()["pos"]
        og = port.geom(n, box, box / scale, scale)
        hi, cse, srt = port.build_cells(og, x, rad)
        assert np.array_equal(s.forces(), psim.force_evaluate(p, g, srt, hi, cse))
    s.close()


@pytest.mark.parametrize("n,box,scale", [(1, 9.0, 5), (257, 9.0, 5), (ORDER_MAX, 45.0, 29),
                                         (ORDER_MAX + 1, 45.0, 29)])
def test_host_arrays_order(psim, n, box, scale):
    rng = np.random.default_rng(n)
    pos, rad = rng.uniform(0.0, box, 3 * n), rng.uniform(0.3, 0.5, n)
    g = psim.geometry(n, box, box / scale, scale)
    hi, cse, srt = port.build_cells(port.geom(n, box, box / scale, scale), pos, rad)
    got = psim.cells_build(g, pos, rad)
    assert np.array_equal(got[0], hi) and np.array_equal(got[2], srt)
    assert np.array_equal(got[1], cse)
    pos[3 * (n // 2)] = box * 1.5
    with pytest.raises(psim.PsimError) as e:
        psim.cells_build(g, pos, rad)
    assert e.value.code == psim.ERR_CELL_BOUNDS


def test_refused_arrays_leave_the_forces_alone(psim):
    n, box, scale = 300, 9.0, 5
    pos, rad = np.random.default_rng(1).uniform(0.0, box, 3 * n), np.full(n, 0.1)
    p = psim.make_force("AO", 1.2, kT=1.0, well_depth=0.3)
    g = psim.geometry(n, box, box / scale, scale)
    hi, cse, srt, ref, err, _ = oracle_force(p.as_dict(), g, pos, rad)
    for bad in (-1, n):
        h = hi.copy()
        h[1] = bad
        out = np.full(3 * n, 7.0)
        with pytest.raises(psim.PsimError) as e:
            psim.force_evaluate(p, g, srt, h, cse, out=out)
        assert e.value.code == psim.ERR_INPUT and np.all(out == 7.0)
