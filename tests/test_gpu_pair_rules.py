"""The FP64 pass where the reference's own rules decide a pair in ways that a shorter
form of them would not: an r^2 whose rounding changes its high word at the cutoff, and
the unit vector's image in a box of edge 1."""
import numpy as np
import pytest

from gpu_helpers import FORCE_TOL_FP64, oracle_force, rel_per_particle

pytestmark = pytest.mark.gpu


def check(psim, g, p, pos, rad):
    hi, cse, srt, ref, err, sc = oracle_force(p.as_dict(), g, pos, rad)
    assert err == 0 and np.any(ref)
    f = psim.force_evaluate(p, g, srt, hi, cse)
    assert rel_per_particle(f, ref, sc) <= FORCE_TOL_FP64


# rc and pairs whose r^2, rounded product by product, is below rc^2 (low word all ones)
# while the one summed with fused multiply-adds has the next high word
TIES = [("0x1.3c26cd02a1a32p+1", ("0x1.9fdec9bae5c8ep-1", "0x1.dba8bde5d4475p+0",
                                  "0x1.68ff26ae177a9p+0")),
        ("0x1.da5e12bfca78ep+0", ("0x1.586fcaf999809p+0", "0x1.f929008cc85abp-1",
                                  "0x1.9cc0a776ad1c7p-1")),
        ("0x1.a712b8c6f54dbp+0", ("0x1.2c92dd0559e41p+0", "0x1.cc3adae5735ddp-1",
                                  "0x1.79daab19d50b3p-1")),
        ("0x1.5478c3667c86cp+1", ("0x1.e1d636145af55p+0", "0x1.8d4ac6502e9fap+0",
                                  "0x1.0f6f104312666p+0"))]


@pytest.mark.parametrize("k", range(len(TIES)))
def test_cutoff_below_a_high_word(psim, force_pass, k):
    rc, d = float.fromhex(TIES[k][0]), [float.fromhex(v) for v in TIES[k][1]]
    assert (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2] < rc * rc
    p = psim.make_force("LJ", rc, kT=1.0, well_depth=1.0, lj_num=6, yukawa_strength=0.0)
    check(psim, psim.geometry(2, 12.0, 3.0, 4), p, np.array([0.0, 0.0, 0.0] + d), np.full(2, 0.5))


@pytest.mark.parametrize("kind", ["LJ6", "LJ9Y", "CAL"])
@pytest.mark.parametrize("box", [1.0, 2.0, 3.0])
def test_unit_vector_in_a_box_of_edge_1(psim, force_pass, kind, box):
    # |d| > int(L)/2 is |d| > 0 in a box of edge 1: the reference's unit vector then
    # points to another image than the one r^2 was taken of
    p = {"LJ6": lambda rc: psim.make_force("LJ", rc, kT=1.0, well_depth=1.0, lj_num=6,
                                           yukawa_strength=0.0),
         "LJ9Y": lambda rc: psim.make_force("LJ", rc, kT=1.0, well_depth=0.5, lj_num=9,
                                            yukawa_strength=1.0, debye_length=0.1),
         "CAL": lambda rc: psim.make_force("CAL", rc)}[kind](0.3 * box)
    rng = np.random.default_rng(0)
    i = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = np.mod(((i + 0.5) * 0.2 + rng.uniform(-0.04, 0.04, i.shape)) * box, box).reshape(-1)
    check(psim, psim.geometry(125, box, box / 3, 3), p, pos, np.full(125, 0.05 * box))


def test_boxes_of_edge_1_in_a_batch_and_a_system(psim):
    # one replica of edge 1 beside one of edge 2, and each alone: the same forces, bit for
    # bit, and the oracle's
    i = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = (i + 0.5) * 0.2 + np.random.default_rng(1).uniform(-0.04, 0.04, i.shape)
    single, reps, pos, rad = [], [], [], []
    for box in (1.0, 2.0):
        p = psim.make_force("LJ", 0.3 * box, kT=1.0, well_depth=1.0, lj_num=6, yukawa_strength=0.0)
        g, r = psim.geometry(125, box, box / 3, 3), np.full(125, 0.05 * box)
        q = np.mod(x * box, box).reshape(-1)
        s = psim.System(g, p, dt=0.001, precision=psim.PRECISION_FP64)
        s.upload(q, r)
        s.step(3)
        f, now = s.forces(), s.download()["pos"]
        s.close()
        *_, ref, err, sc = oracle_force(p.as_dict(), g, now, r)
        assert err == 0 and rel_per_particle(f, ref, sc) <= FORCE_TOL_FP64
        single.append(f)
        reps.append((g, p))
        pos.append(q)
        rad.append(r)
    b = psim.Batch([(g, p, 90210) for g, p in reps], dt=0.001,
                   precision=psim.PRECISION_FP64)
    b.upload(np.concatenate(pos), np.concatenate(rad))
    b.step(3)
    assert np.array_equal(b.forces(), np.concatenate(single))
    b.close()
