"""The integer-grid arithmetic of the FP64 step (fixed64.cuh, collide64.cuh), compiled for the host, against
exact rationals."""
import ctypes
import os
import subprocess
from fractions import Fraction as F

import numpy as np
import pytest

from conftest import PKG, REPO


@pytest.fixture(scope="module")
def fxh(tmp_path_factory):
    import rbtp_build
    try:
        nvcc = rbtp_build.nvcc()
    except RuntimeError as e:
        pytest.skip(str(e))
    lib = tmp_path_factory.mktemp("fx") / "libfxh.so"
    subprocess.run([nvcc, *rbtp_build.ARCH, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-shared",
                    "-Xcompiler", "-fPIC,-ffp-contract=off", "-I" + os.path.join(PKG, "csrc"),
                    "-I" + os.path.join(REPO, "include"), os.path.join(REPO, "tests", "fx_host.cu"), "-o", str(lib)],
                   check=True)
    return ctypes.CDLL(str(lib))


def test_a_sixth_of_the_squared_velocity_has_no_one_sided_error(fxh):
    """sum_i w_i ((c_i.v)^2 / 2 - v^2 / 6) vanishes only if the rounding of v^2 / 6 is a matter of chance.  Two
    sums and a product round by at most 2^-53 each, so a mean over n samples lies within 5 * 3 * 2^-53 / sqrt(n)."""
    n, rng, out = 20000, np.random.default_rng(1), (ctypes.c_double * 4)()
    total = F(0)
    for u in 0.1 * rng.uniform(-1, 1, (n, 3)):
        fxh.fxh_vel((ctypes.c_double * 3)(*u), out)
        want = F(out[1]) + F(out[2]) + F(out[3])
        total += (6 * F(out[0]) - want) / want
    assert abs(float(total / n)) < 5 * 3 * 2.0 ** -53 / n ** 0.5
