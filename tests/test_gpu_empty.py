"""Systems and host arrays without particles, in each form: nothing to do, and the step
count goes on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NONE = np.zeros(0)


@pytest.mark.parametrize("precision,skin", [(0, 0.0), (1, 0.0), (1, 0.3)])
def test_steps_of_an_empty_system(psim, precision, skin):
    g = psim.geometry(0, 12.0, 1.5, 8)
    s = psim.System(g, psim.make_force("AO", 1.1, kT=1.0, well_depth=0.25), vel_freq=3,
                    precision=precision, skin=skin)
    s.upload(NONE, NONE)
    for k in (1, 5, 30):
        s.step(k)
    assert s.get_step() == (36, 35 % 4)
    s.profile(2)
    assert s.get_step()[0] == 38 and s.list_builds() == 0
    assert s.download()["pos"].size == 0 and s.forces().size == 0
    assert s.energy() == (0.0, 0.0) and s.temperature() == 0.0
    assert s.clusters(1.2, 4)[1] == []
    s.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_drop_ins_without_particles(psim, precision):
    g = psim.geometry(0, 12.0, 1.5, 8)
    hi, cse, srt = psim.cells_build(g, NONE, NONE)
    assert hi.size == 0 and srt.size == 0 and np.all(cse == 0xffffffff)
    f = psim.force_evaluate(psim.make_force("AO", 1.1, kT=1.0, well_depth=0.25), g, srt, hi, cse,
                            precision=precision)
    assert f.size == 0
