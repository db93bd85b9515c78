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
    L = ctypes.CDLL(str(lib))
    D, U, I, LL = ctypes.c_double, ctypes.c_uint, ctypes.c_int, ctypes.c_longlong
    for name, res, args in (("grid", U, [D]), ("from", LL, [D, U]), ("to", D, [LL, U, I]), ("times", LL, [D, D, U, I]),
                            ("choice", I, [LL, LL])):
        fn = getattr(L, "fxh_" + name)
        fn.restype, fn.argtypes = res, args
    return L


def _unit(grid, up=0):
    """The value of one unit of a grid, times 2^up."""
    return F(2) ** ((grid >> 20) - 1075 - 5 + up)


def _doubles(rng, n, below):
    """n doubles 2^0 to 2^-below of 1, of all significands, some with few bits, of both signs, and zeros."""
    bits = rng.choice([53, 53, 20, 3, 1], n)
    m = [int(rng.integers(0, 2 ** 53)) >> (53 - int(b)) << (53 - int(b)) for b in bits]
    return [float(rng.choice([-1, 1])) * (1 + k / 2 ** 53) * 2.0 ** -int(rng.integers(0, below + 1)) if k % 31 else 0.0
            for k in m]


def _odd(d, unit):
    """d / unit rounded to odd: towards zero, and the last place set if a one was cut off (looked for in the low
    word of the significand); what is below 1 becomes 0."""
    x = abs(F(d) / unit)
    n = x.numerator // x.denominator
    low_word = int(np.array(d).view(np.uint64)) & 0xffffffff
    n |= n % 2 ** 32 != 0 and x.denominator > 1 and low_word != 0
    return n if d > 0 else -n


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


def test_members_are_rounded_to_odd_on_the_grid(fxh):
    rng = np.random.default_rng(2)
    for scale in (1.0, 2.0 ** -40, 2.0 ** 14):
        grid = fxh.fxh_grid(scale * 1.5)
        for d in _doubles(rng, 6000, 75):
            assert fxh.fxh_from(scale * d, grid) == _odd(scale * d, _unit(grid)), d.hex()


def test_sums_are_rounded_to_nearest_even_doubles(fxh):
    rng = np.random.default_rng(3)
    grid = fxh.fxh_grid(0.3)
    for k in range(12000):
        v = int(rng.integers(-2 ** 63 + 1, 2 ** 63)) >> int(rng.integers(0, 63))
        v = v >> 9 << 9 if k % 3 == 0 else v   # ties
        assert fxh.fxh_to(v, grid, -1 - k % 5) == float(v * _unit(grid, -1 - k % 5)), v


def test_products_are_rounded_to_odd_on_the_grid(fxh):
    """The 64-bit product lies up to 3 of its last places below the exact one, and at least 2 places are cut
    off it, so the result is within two units; from two units on it favours no side on average: the mean stays
    within four deviations (a third of a unit's square), and the 3 places in the few largest."""
    rng = np.random.default_rng(4)
    grid, total, n = fxh.fxh_grid(1.0), F(0), 0
    for j, d in enumerate(_doubles(rng, 24000, 40)):
        k = (-0.5, 0.0)[j % 2] if j < 4000 else float(rng.uniform(-1, 1))
        got, want = fxh.fxh_times(k, d, grid, 5), F(k) * F(d) / _unit(grid, 5)
        assert abs(got - want) < 2 and (got != 0 or abs(want) < 1.001)
        if j >= 4000 and abs(want) >= 2:
            total += (got - want) * (1 if want > 0 else -1)
            n += 1
    assert abs(float(total / n)) < 4 * 3 ** -0.5 / n ** 0.5 + 2.0 ** -8


@pytest.mark.parametrize("sms", [76, 132, 148, 152, 160])
def test_variant_of_a_grid_follows_the_multiprocessor_count(fxh, sms):
    """Four waves of nine resident blocks are the last unrolled grid; twelve are taken where ceil(blocks / 12 sms)
    is below the waves of nine, of which the last counts from a quarter on."""
    for blocks in [1, sms, *(k * sms * n + d for n in (9, 12) for k in (1, 2, 3, 4, 5) for d in (-1, 0, 1, 2 * sms, 3 * sms)), 10 ** 6]:
        waves = -(-(blocks - 9 * sms // 4) // (9 * sms))
        unrolled = blocks <= 36 * sms
        most = unrolled and -(-blocks // (12 * sms)) < waves
        assert fxh.fxh_choice(blocks, sms) == unrolled + 2 * most, blocks
