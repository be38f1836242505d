"""The FP64 passes' own 1/a, 1/sqrt(a), sqrt(a) and exp(x) against extended precision and beside
CUDA's, over the ranges of their arguments, in units of 2^-53 of the value.

Bounds.  The last operation of each rounds once: at most 1, and 0.4247 in the mean square
(uniform in the last place, 1/mantissa^2 averaged over a logarithmic range).
1/a: the seed's error cubed beside it, below 0.07 for a seed of 19 bits.
1/sqrt(a): half the rounding of a y as well, 0.5 at most and sqrt(0.4247^2 + 0.2124^2) =
0.4748 in all, and 5/16 of the seed's error cubed.
exp(x): what the cubic coefficient leaves of r^5/120, 0.045 at |r| = ln2/512, and the
roundings of a term of 1.4e-3 of the value."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

N = 1 << 20
ULP = np.longdouble(2) ** -53


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from proteinsim2015_gb300 import build
    so = str(tmp_path_factory.mktemp("math") / "fp64_math.so")
    subprocess.check_call([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-shared",
                           "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I", build.CSRC,
                           os.path.join(ROOT, "tests", "kernels", "fp64_math.cu"), "-o", so])
    lib = C.CDLL(so)
    lib.run.argtypes = [C.c_int, C.c_int, C.c_void_p, C.c_void_p]

    def call(what, x):
        out = np.empty_like(x)
        assert lib.run(what, len(x), x.ctypes.data, out.ctypes.data) == 0
        return out
    return call


def errors(got, want):
    e = (got.astype(np.longdouble) / want - 1) / ULP
    return float(np.max(np.abs(e))), float(np.sqrt(np.mean(e * e)))


CASES = {   # number, range (of the exponent of 2, or of x), largest and rms error
    "rcp_pairs": (0, (-14, 14), 1.07, 0.43),
    "rcp_wide": (0, (-1000, 1000), 1.07, 0.43),
    "rsqrt_pairs": (2, (-14, 14), 1.53, 0.48),
    "rsqrt_wide": (2, (-1000, 1000), 1.53, 0.48),
    "exp_pairs": (4, (-14.0, 0.0), 1.06, 0.43),
    "exp_wide": (4, (-689.0, 689.0), 1.06, 0.43),
}


@pytest.mark.parametrize("name", list(CASES))
def test_errors(run, name):
    assert np.finfo(np.longdouble).nmant >= 63
    what, (lo, hi), most, rms = CASES[name]
    rng = np.random.default_rng(11)
    if what == 4:
        x = rng.uniform(lo, hi, N)
        want = np.exp(x.astype(np.longdouble))
    else:
        x = np.ldexp(2.0 ** rng.uniform(0.0, 1.0, N), rng.integers(lo, hi, N).astype(np.int32))
        a = x.astype(np.longdouble)
        want = 1 / a if what == 0 else 1 / np.sqrt(a)
    ours, cuda = errors(run(what, x), want), errors(run(what + 1, x), want)
    print(name, "largest, rms: %.3f %.4f" % ours, "CUDA's: %.3f %.4f" % cuda)
    assert ours[0] <= most and ours[1] <= rms
    assert ours[1] <= 1.005 * cuda[1]    # sampling: 1 / sqrt(2 N) = 0.07%
    if what > 0:                         # (1/a is rounded correctly by CUDA)
        assert ours[0] <= cuda[0]


def test_exp_edges(run):
    x = np.array([0.0, -0.0, -690.0, 690.0, -700.0, -745.2, -1e6, 700.0, 709.8, np.inf, -np.inf,
                  np.nan, 1e-300, -1e-300, 5e-324])
    ours, cuda = run(4, x), run(5, x)
    assert np.array_equal(ours, cuda, equal_nan=True)


@pytest.mark.parametrize("lo,hi", [(-14, 14), (-1000, 1000)])
def test_sqrt_is_correctly_rounded(run, lo, hi):
    rng = np.random.default_rng(12)
    x = np.ldexp(2.0 ** rng.uniform(0.0, 1.0, N), rng.integers(lo, hi, N).astype(np.int32))
    assert np.array_equal(run(6, x), np.sqrt(x))
