"""step_async does not wait for the device, whatever phase and kind of step a call in the
middle of a run is the first to reach."""
import numpy as np
import pytest

from gpu_helpers import rsa_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vel_freq", [0, 1, 2, 25])
@pytest.mark.parametrize("precision,skin", [(0, 0.0), (1, 0.0), (1, 0.3)])
@pytest.mark.parametrize("first", [1, 4])
def test_later_steps_are_enqueued_at_once(psim, precision, skin, vel_freq, first):
    import torch
    n, box = 400, 12.0
    pos, rad = rsa_state(n, box, seed=8)
    s = psim.System(psim.geometry(n, box, 1.5, 8), psim.make_force("AO", 1.1, kT=1.0,
                                                                   well_depth=0.25),
                    gamma=1.0, dt=0.001, kT=1.0, vel_freq=vel_freq, seed=5, precision=precision,
                    skin=skin)
    s.upload(pos, rad, vel=np.random.default_rng(8).standard_normal(3 * n))
    s.step(first)
    stream, busy = torch.cuda.ExternalStream(s.stream()), torch.cuda.Event()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(300_000_000)   # ~0.15 s of the stream
        busy.record()
    for k in (1, 1, 1, 1, 1, 1, 7):
        s.step_async(k)
    waited = busy.query()
    s.sync()
    assert not waited and s.get_step()[0] == first + 13
    s.close()


@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
@pytest.mark.parametrize("vel_freq", [0, 12, 25])
@pytest.mark.parametrize("precision,skin", [(0, 0.0), (1, 0.0), (1, 0.3)])
def test_a_callers_capture_is_refused(psim, precision, skin, vel_freq):
    # whatever kind of step comes first in it; the system goes on afterwards
    import torch
    n, box = 400, 12.0
    pos, rad = rsa_state(n, box, seed=8)
    s = psim.System(psim.geometry(n, box, 1.5, 8), psim.make_force("AO", 1.1, kT=1.0,
                                                                   well_depth=0.25),
                    gamma=1.0, dt=0.001, kT=1.0, vel_freq=vel_freq, seed=5, precision=precision,
                    skin=skin)
    s.upload(pos, rad)
    s.step(1)
    stream = torch.cuda.ExternalStream(s.stream())
    for k in range(15):      # steps 1 to 15: a velocity step among them where vel_freq is 12
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream,
                              capture_error_mode="thread_local"):
            with pytest.raises(psim.PsimError):
                s.step_async(1)
        s.step(1)
    assert s.get_step()[0] == 16
    s.close()
