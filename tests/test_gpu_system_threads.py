"""One resident system read by several threads at once: each call's answer is the one it
gives alone, whatever scratch the others take meanwhile."""
import threading

import numpy as np
import pytest

from proteinsim2015_gb300 import init

pytestmark = pytest.mark.gpu


def flat(v):
    if isinstance(v, dict):
        return [np.asarray(x) for _, x in sorted(v.items())]
    if isinstance(v, (list, tuple)):
        return [np.asarray(y) for x in v for y in flat(x)]
    return [np.asarray(v)]


@pytest.mark.parametrize("precision,skin", [(0, 0.0), (1, 0.0), (1, 0.3)])
def test_reads_from_several_threads(psim, precision, skin):
    n, box = 20000, 42.0
    g = psim.geometry(n, box, 1.5, 28)
    pos = init.rsa_native(n, box, 1.0, seed=4).reshape(-1)
    s = psim.System(g, psim.make_force("AO", 1.1, kT=1.0, well_depth=0.25), dt=0.001, vel_freq=5,
                    precision=precision, skin=skin)
    s.upload(pos, np.full(n, 0.5), vel=init.maxwell(n, 1.0, seed=4).reshape(-1))
    s.step(13)
    calls = [s.download, s.download_cells, s.forces, s.temperature, s.mean_displacement, s.energy,
             lambda: s.interactions(1.2), lambda: s.rdf(0.8, 1.5, 50),
             lambda: s.clusters(1.2, 4), lambda: s.pair_count(1.1), s.cell_occupancy]
    want = [flat(c()) for c in calls]
    wrong = []

    def work(k):
        try:
            for r in range(3 * len(calls)):
                c = (k * 5 + r) % len(calls)
                got = flat(calls[c]())
                if len(got) != len(want[c]) or not all(
                        np.array_equal(a, b) for a, b in zip(got, want[c])):
                    wrong.append(c)
        except Exception as e:   # noqa: BLE001 -- reported below, with the thread's number
            wrong.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    s.close()
    assert not wrong
