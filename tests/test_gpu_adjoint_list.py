"""The adjoint's neighbour list: particles that leave it inside a segment (steps
taken again on a new list), each number of lanes a particle, bins beyond shared
memory, and the same bits from two runs.  Gradients against FP64 forward-mode
tangents on the CPU (the adjoint's own tolerance) and central differences."""
import numpy as np
import pytest

from test_gpu_adjoint import _lj_params, setup

pytestmark = pytest.mark.gpu


def against_tangent(psim, oracle_port, speed, T, every, K, nb, seed=31):
    from proteinsim2015_gb300 import adjoint as adj
    g, pos, vel = setup(psim, seed=95)
    vel = vel * speed
    p, _ = adj.plugin_params(3.0, 0.1, 10.0, 4.0)
    p.ao_cutoff = 0.0        # the soft Yukawa repulsion alone
    pt = adj.AdjointParams.from_buffer_copy(p)
    pt.yuk_amplitude *= 1.3
    a = adj.Adjoint(g, T, dt=0.001, seed=seed, checkpoint_every=K, sample_every=every, n_bins=nb)
    target = a.forward(pt, pos, vel)
    loss, gm, grad, gp = a.gradient(p, pos, target, vel, wrt_pos=True)
    a.close()
    noise = psim.philox_noise(seed, g.n_particles, 0, T)
    tl, tg, tgrad = oracle_port.adjoint_tangent(g.box_size, p, 1.0, 0.001, 1.0, 1.0, T, every, 0.8,
                                                3.0, nb, 2.2 / nb, pos, vel, noise, target)
    assert loss == pytest.approx(tl, rel=1e-9)
    assert np.allclose(gm, tg, rtol=1e-9, atol=1e-12)
    for k in (2, 3):         # Yukawa amplitude and length
        assert grad[k] == pytest.approx(tgrad[k], rel=1e-6, abs=1e-9 * max(abs(tgrad)))
    assert np.all(np.isfinite(gp))


@pytest.mark.parametrize("K", [2, 16, 40])
def test_particles_that_leave_the_list(psim, oracle_port, K):
    # speeds of ~35: half the skin in about two steps
    against_tangent(psim, oracle_port, 20.0, 40, 4, K, 60)


def test_bins_beyond_shared_memory(psim, oracle_port):
    against_tangent(psim, oracle_port, 1.0, 12, 3, 5, 3100)


@pytest.mark.parametrize("n", [4096, 4097, 12287, 12288])   # 16, 8, 8 and 4 lanes
def test_lanes(psim, n):
    from proteinsim2015_gb300 import adjoint as adj
    from proteinsim2015_gb300 import init
    import math
    box = (n * math.pi / 6.0 / 0.15) ** (1.0 / 3.0)
    scale = int(box // 3.1)
    g = psim.geometry(n, box, box / scale, scale)
    pos = init.rsa_native(n, box, 1.0, seed=n).reshape(-1)
    vel = init.maxwell(n, 1.0, seed=n).reshape(-1)
    a = adj.Adjoint(g, 20, dt=0.001, seed=3, checkpoint_every=8, sample_every=5)
    p, _ = _lj_params(adj)
    target = np.ones(100)
    loss, gm, grad, gp = a.gradient(p, pos, target, vel, wrt_pos=True)
    again = a.gradient(p, pos, target, vel, wrt_pos=True)
    assert again[0] == loss and np.array_equal(again[1], gm)
    assert np.array_equal(again[2], grad) and np.array_equal(again[3], gp)
    for k, name in ((2, "yuk_amplitude"), (3, "yuk_length")):
        h = 1e-5 * getattr(p, name)
        qp, qm = adj.AdjointParams.from_buffer_copy(p), adj.AdjointParams.from_buffer_copy(p)
        setattr(qp, name, getattr(p, name) + h)
        setattr(qm, name, getattr(p, name) - h)
        fd = (np.sum((a.forward(qp, pos, vel) - target) ** 2) -
              np.sum((a.forward(qm, pos, vel) - target) ** 2)) / (2 * h)
        assert grad[k] == pytest.approx(fd, rel=1e-3), name
    a.close()
