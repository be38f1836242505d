"""The FP64 force pass at the sizes where its walk changes: a warp's eight
particles, a queue that is drained several times, a row of cells per lane
against a row at a time, unequal radii, and pairs next to the cutoff and the
overlap distance, where the reference's own rounding of r^2 decides.  Forces
within 1e-12 of sum_j |f_ij| of the oracle (the plain form's tolerance)."""
import numpy as np
import pytest

from gpu_helpers import FORCE_TOL_FP64, lattice_state, oracle_force, rel_per_particle
from oracle import port

pytestmark = pytest.mark.gpu


def check(psim, g, p, pos, rad):
    hi, cse, srt, ref, err, sc = oracle_force(p.as_dict(), g, pos, rad)
    assert err == 0
    f = psim.force_evaluate(p, g, srt, hi, cse)
    assert rel_per_particle(f, ref, sc) <= FORCE_TOL_FP64
    return f


def forces_of(psim, kind):
    if kind == "LJ5":      # odd exponent, no Yukawa term
        return psim.make_force("LJ", 2.5, kT=1.2, well_depth=0.7, lj_num=5, yukawa_strength=0.0)
    if kind == "LJ12Y":
        return psim.make_force("LJ", 2.5, kT=1.0, well_depth=2.0, lj_num=12, yukawa_strength=4.0)
    if kind == "AO_YUK":
        return psim.make_force("AO_YUK", 1.1, well_depth=0.2, cutoff2=2.5, well_depth2=1.0,
                               yukawa_strength=50.0, debye_length=0.3, lj_num=0)
    if kind == "CAL":
        return psim.make_force("CAL", 1.5)
    return psim.make_force("AO", 1.3, well_depth=0.5)


@pytest.mark.parametrize("kind", ["LJ5", "LJ12Y", "AO_YUK", "CAL", "AO"])
@pytest.mark.parametrize("n,scale", [(1, 4), (7, 4), (9, 4), (500, 4), (499, 3), (255, 4)])
def test_walk_edges(psim, kind, n, scale):
    # up to 7.8 (scale 4: a row per lane) and 18.5 particles a cell (scale 3)
    pos, _, box = lattice_state(5, 2.4, 0.3, seed=n)
    keep = np.sort(np.random.default_rng(n).permutation(500)[:n])
    pos = pos.reshape(-1, 3)[keep].reshape(-1)
    rad = np.random.default_rng(n + 1).uniform(0.3, 0.55, n)
    check(psim, psim.geometry(n, box, box / scale, scale), forces_of(psim, kind), pos, rad)


def test_queue_drained_several_times(psim):
    # ~460 neighbours a particle, against 128 queue entries
    pos, rad, box = lattice_state(9, 4.0 / 3.0, 0.05, seed=3)
    rad[:] = 0.3
    p = psim.make_force("LJ", 4.0, kT=1.0, well_depth=1.0, lj_num=6, yukawa_strength=0.0)
    check(psim, psim.geometry(len(rad), box, box / 3, 3), p, pos, rad)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("x0", [3.0, 11.3])   # inside the box, across its edge
def test_cutoff_is_decided_as_the_reference_does(psim, axis, x0):
    box, rc = 12.0, 2.5
    g = psim.geometry(2, box, 3.0, 4)
    p = psim.make_force("LJ", rc, kT=1.0, well_depth=1.0, lj_num=6, yukawa_strength=0.0)
    rng = np.random.default_rng(5)
    seen = set()
    for _ in range(40):
        a = np.array([6.1, 6.2, 6.3])
        a[axis] = x0
        d = rng.normal(size=3)
        d[axis] = abs(d[axis]) + 2.0
        b = a + d * (rc / np.linalg.norm(d)) * (1.0 + rng.integers(-2, 3) * 2.0 ** -53)
        pos = np.mod(np.concatenate([a, b]), box)
        f = check(psim, g, p, pos, np.full(2, 0.5))
        seen.add(bool(np.any(f)))
    assert seen == {True, False}


@pytest.mark.parametrize("ulps", [-2, -1, 0, 1, 2])
def test_overlap_is_decided_as_the_reference_does(psim, ulps):
    g = psim.geometry(2, 12.0, 3.0, 4)
    r = 0.8 * (0.45 + 0.55)
    for _ in range(abs(ulps)):
        r = np.nextafter(r, 0.0 if ulps < 0 else 1.0)
    for rad in (np.array([0.45, 0.55]), np.array([0.5, 0.5])):
        pos = np.array([1.0, 0.25, 1.0, 1.0, 0.25 + r, 1.0])
        p = psim.make_force("CAL", 1.5)
        og = port.geom(2, 12.0, 3.0, 4)
        hi, cse, srt = port.build_cells(og, pos, rad)
        _, err = port.forces(og, port.force_from_params(p.as_dict()), srt, hi, cse)
        if err:
            with pytest.raises(psim.PsimError) as e:
                psim.force_evaluate(p, g, srt, hi, cse)
            assert e.value.code == psim.ERR_OVERLAP
        else:
            psim.force_evaluate(p, g, srt, hi, cse)
