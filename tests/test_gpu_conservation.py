"""Mass of a closed box over many FP64 steps.  Collisions, bounce-back and streaming keep sum f; what is left is
the rounding of each collided population, which must be a matter of chance.  A population takes some four
roundings of at most 2^-53 of itself, so sum f after n steps lies within 6 * 4 * 2^-53 * rms(f) * sqrt(27 L n)."""
import math

import numpy as np
import pytest

from rbtp import Solver, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lx,ly,lz,ra", [(16, 12, 8, 2e4), (16, 12, 8, 1e5), (35, 10, 6, 1e5)])
def test_mass_of_a_closed_box_does_not_drift(lib_built, lx, ly, lz, ra):
    steps, cfg = 20000, W.config("plain_fp64", lx=lx, ly=ly, lz=lz, rayleigh=ra)
    s = Solver(cfg)
    s.load_state(*W.initial_state(cfg, seed=2, amp=5e-2))
    s.step(2000)
    before = math.fsum(s.fg()[0])
    s.step(steps)
    f = s.fg()[0]
    rms = float(np.sqrt(np.mean(f * f)))
    assert rms > 1e-5   # the fluid moves
    assert abs(math.fsum(f) - before) < 6 * 4 * 2.0 ** -53 * rms * math.sqrt(27 * cfg.nodes * steps)
