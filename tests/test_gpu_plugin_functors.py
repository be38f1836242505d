"""Plugins whose pair functor is built on one of the library's: the force is the
functor's own in both precisions, as its CPU getAcceleration gives it, against the
oracle."""
import os

import numpy as np
import pytest

from conftest import ROOT
from gpu_helpers import FORCE_TOL_FP64, FORCE_TOL_MIXED, oracle_force, rel_norm, rel_per_particle
from proteinsim2015_gb300 import init

pytestmark = pytest.mark.gpu

N, BOX, SCALE = 1500, 24.0, 8
SETTINGS = dict(kT=1.3, wellDepth=0.9, cutOff=2.5, debyeLength=0.4)


@pytest.fixture(scope="module")
def plugin_so(psim, tmp_path_factory):
    from proteinsim2015_gb300 import build
    return build.build_force_plugin(os.path.join(ROOT, "tests", "plugins", "functor_plugin.cu"),
                                    out=str(tmp_path_factory.mktemp("functor") / "Functor.so"),
                                    include_dirs=[build.CSRC])


def check(psim, plugin_so, settings, lj_num, yukawa):
    """The plugin with these settings against LJ(lj_num) with that Yukawa strength."""
    text = "".join("%s = %r\n" % kv for kv in dict(SETTINGS, **settings).items())
    plug = psim.ForcePlugin(plugin_so, "force = Functor\n" + text)
    want_p = psim.make_force("LJ", SETTINGS["cutOff"], kT=SETTINGS["kT"],
                             well_depth=SETTINGS["wellDepth"], lj_num=lj_num,
                             yukawa_strength=yukawa, debye_length=SETTINGS["debyeLength"])
    g = psim.geometry(N, BOX, BOX / SCALE, SCALE)
    pos, rad = init.rsa(N, BOX, 1.0, seed=21).reshape(-1), np.full(N, 0.5)
    hi, cse, srt, want, err, scale = oracle_force(want_p.as_dict(), g, pos, rad)
    assert err == 0
    got = psim.force_evaluate(plug, g, srt, hi, cse, precision=psim.PRECISION_FP64)
    assert rel_per_particle(got, want, scale) <= FORCE_TOL_FP64
    got = psim.force_evaluate(plug, g, srt, hi, cse, precision=psim.PRECISION_MIXED)
    assert rel_norm(got, want) <= FORCE_TOL_MIXED


@pytest.mark.parametrize("lj_num", [6, 7])
def test_derived_functor_keeps_its_own_force(psim, plugin_so, lj_num):
    check(psim, plugin_so, dict(variant=0, ljNum=lj_num, yukawaStrength=3.0), 0, 3.0)


@pytest.mark.parametrize("variant", [1, 2])
@pytest.mark.parametrize("lj_num,yukawa", [(6, 3.0), (7, 3.0), (6, 0.0)])
def test_functor_filled_by_the_plugin(psim, plugin_so, variant, lj_num, yukawa):
    check(psim, plugin_so, dict(variant=variant, ljNum=lj_num, yukawaStrength=yukawa), lj_num,
          yukawa)
