"""The pair observables at the edges of their walk: fewer particles than a warp
takes, grids of three cells a side, and both ways a warp takes its rows, against
sums over all pairs in numpy."""
import numpy as np
import pytest

from gpu_helpers import lattice_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,scale", [(1, 3), (2, 3), (9, 3), (17, 8), (499, 3), (500, 8)])
@pytest.mark.parametrize("precision,skin", [(0, 0.0), (1, 0.0), (1, 0.05)])
def test_pair_observables(psim, n, scale, precision, skin):
    pos, _, box = lattice_state(5, 2.0, 0.2, seed=n + scale)
    keep = np.sort(np.random.default_rng(n).permutation(500)[:n])
    pos = pos.reshape(-1, 3)[keep]
    p = psim.make_force("AO", 1.15, kT=1.0, well_depth=0.5)
    s = psim.System(psim.geometry(n, box, box / scale, scale), p, precision=precision, skin=skin)
    s.upload(pos.reshape(-1), np.full(n, 0.3))
    i, j = np.triu_indices(n, 1)
    d = pos[j] - pos[i]
    d -= box * np.round(d / box)
    r = np.linalg.norm(d, axis=1)
    c1, c2 = psim.ao_coefficients(1.0, 0.5, 1.15)
    q = r[r < 1.15]
    u = 36 / 37 * (q ** -37 - 1.15 ** -37) + c1 * np.log(1.15 / q) + 0.5 * c2 * (1.15 ** 2 - q * q)
    w = (36 * q ** -38 + c1 / q + c2 * q) * q
    e = s.energy()
    assert e[0] == pytest.approx(u.sum() / n, rel=1e-11, abs=1e-13)
    assert e[1] == pytest.approx(w.sum() / n, rel=1e-11, abs=1e-13)
    near = r < 1.2
    coor, total = s.interactions(1.2)
    assert np.array_equal(coor, np.bincount(np.concatenate([i[near], j[near]]), minlength=n))
    assert total == 2 * near.sum()
    g = s.rdf(0.5, 1.25, 30)
    h = np.histogram(r, 30, (0.5, 1.25))[0]
    edge = np.linspace(0.5, 1.25, 31)
    shell = 4 / 3 * np.pi * (edge[1:] ** 3 - edge[:-1] ** 3)
    assert np.allclose(g, 2 * h / (n * n / box ** 3 * shell), rtol=1e-12)
    root, groups, _ = s.clusters(1.2, 1)
    label = np.arange(n)
    for _ in range(n):
        low = np.minimum(label[i[near]], label[j[near]])
        new = label.copy()
        np.minimum.at(new, i[near], low)
        np.minimum.at(new, j[near], low)
        if np.array_equal(new, label):
            break
        label = new
    assert np.array_equal(root, label)
    want = [np.flatnonzero(label == k) for k in range(n) if np.sum(label == k) > 1]
    assert len(groups) == len(want) and all(np.array_equal(a, b) for a, b in zip(groups, want))
    s.close()
