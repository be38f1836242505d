"""Bins on both sides of what the smoothed counts hold in shared memory, for each
number of lanes a particle: one step, sampled, against the same counts on the CPU."""
import math

import numpy as np
import pytest

from proteinsim2015_gb300 import init

pytestmark = pytest.mark.gpu


def smoothed_g(x, box, r_min, dr, nb, sigma, real=np.float64):
    """Gaussian-smoothed g(r): each pair adds to the bins within its reach."""
    from scipy.spatial import cKDTree
    x = np.mod(x.reshape(-1, 3), box)
    n, reach = len(x), int(math.ceil(4.0 * sigma / dr)) + 1
    i, j = cKDTree(x.astype(np.float64), boxsize=box).query_pairs(r_min + nb * dr + 4.0 * sigma,
                                               output_type="ndarray").T
    d = x[j] - x[i]
    r = np.linalg.norm(d - box * np.round(d / box), axis=1)
    b0, h = np.floor((r - r_min) / dr).astype(np.int64), np.zeros(nb, real)
    for k in range(-reach, reach + 1):
        b = b0 + k
        ok = (b >= 0) & (b < nb)
        z = (r[ok] - (r_min + (b[ok].astype(real) + real(0.5)) * dr)) / sigma
        np.add.at(h, b[ok], 2.0 * dr * np.exp(-0.5 * z * z) / (np.sqrt(real(2.0 * math.pi)) * sigma))
    rb = r_min + (np.arange(nb, dtype=real) + real(0.5)) * dr
    return h / (n * (n / real(box) ** 3) * 4.0 * math.pi * rb * rb * dr)


@pytest.mark.parametrize("n,nb", [(n, nb) for n in (300, 8000, 12288)   # 16, 8 and 4 lanes
                                  for nb in (2944, 2945, 3072, 3073, 5000)])
def test_bins(psim, n, nb):
    from proteinsim2015_gb300 import adjoint as adj
    box = (n * math.pi / 6.0 / 0.15) ** (1.0 / 3.0)
    scale = int(box // 3.1)
    g = psim.geometry(n, box, box / scale, scale)
    pos = init.rsa_native(n, box, 1.0, seed=n).reshape(-1)
    vel = init.maxwell(n, 1.0, seed=n).reshape(-1)
    p, _ = adj.plugin_params(3.0, 0.1, 10.0, 4.0)
    p.ao_cutoff = 0.0        # the soft Yukawa repulsion alone
    a = adj.Adjoint(g, 1, dt=0.001, seed=3, checkpoint_every=2, sample_every=1, n_bins=nb)
    gm, x = a.forward(p, pos, vel, final=True)
    loss, gm2, grad, _ = a.gradient(p, pos, np.ones(nb), vel)
    a.close()
    want = smoothed_g(x, box, 0.8, 2.2 / nb, nb, 2.2 / nb)
    # x is rounded to an ulp of the box (7e-15) where the counts saw it wrapped: z is off
    # by 2e-11 and a term by 1e-10 of itself
    assert np.max(np.abs(gm - want)) <= 1e-9 * max(1.0, np.max(want))
    assert loss == pytest.approx(np.sum((gm2 - 1.0) ** 2), rel=1e-12)
    assert np.all(np.isfinite(grad))


@pytest.mark.parametrize("n", [300, 8000, 12288])
@pytest.mark.parametrize("nb,width", [(100, 1.0), (100, 0.3), (400, 1.0)])
def test_tails_of_the_kernel(psim, n, nb, width):
    # bins that only the tails of a few kernels reach, down to e^-37 of one: each to its own
    # precision.  Particles away from the faces, so that the positions come back as they were.
    from proteinsim2015_gb300 import adjoint as adj
    ld, dr = np.longdouble, (3.0 - 0.8) / nb
    box = (n * math.pi / 6.0 / 0.15) ** (1.0 / 3.0)
    pos = init.rsa_native(n, box, 1.0, seed=n).reshape(-1, 3)
    pos = pos[np.all((pos > 0.02) & (pos < box - 0.02), axis=1)]
    scale = int(box // 3.2)
    p, _ = adj.plugin_params(3.0, 0.1, 10.0, 4.0)
    p.ao_cutoff = 0.0
    a = adj.Adjoint(psim.geometry(len(pos), box, box / scale, scale), 1, dt=0.001, seed=3,
                    checkpoint_every=2, sample_every=1, n_bins=nb, sigma=width * dr)
    g, x = a.forward(p, pos.reshape(-1), final=True)
    g2 = a.forward(p, pos.reshape(-1))
    a.close()
    assert np.array_equal(g, g2)
    assert np.all((x > 0.0) & (x < box))
    want = smoothed_g(x.astype(ld), box, 0.8, dr, nb, width * dr, real=ld)
    some = want > 0
    # r and the bins' centres to 2^-53 of 3: z = (r - r_b) / sigma to 6.7e-16 / sigma, and a
    # term to z = dz (reach + 1/2) <= 25 of these, 2.6e-12 at the narrowest; the rest is less
    assert np.max(np.abs(g[some] / want[some] - 1)) <= 5e-12
    assert np.all(g[~some] == 0)
