"""The solid flags of a step are marked on an array that one kernel clears four nodes at a time: node
counts that are not a multiple of four, and flags that a moving sphere leaves behind."""
import numpy as np
import pytest

from rbtp import Batch, Solver, derive, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lx,ly,lz", [(45, 43, 23), (42, 43, 23), (45, 43, 25)])   # 1, 2 and 3 nodes left over
def test_flags_follow_the_spheres(lib_built, oracle_mod, lx, ly, lz):
    cfg = W.config("plain_fp64", lx=lx, ly=ly, lz=lz, activate_particles=1, particle_diam_frac=8.0 / lx,
                   particle_fraction=0.04, rho_particle_ratio=1.0)
    n = derive(cfg).npart
    o = oracle_mod.Oracle(cfg)
    o.initialize()
    p = o.particles()
    p[:, 3:6] = 0.08 * np.random.default_rng(lx + lz).standard_normal((n, 3))
    state = (*W.initial_state(cfg, seed=3, amp=1e-2), p)
    o.load_state(*state)
    single, member = Solver(cfg), Solver(cfg)
    single.load_state(*state)
    member.load_state(*state)
    b = Batch(0)
    b.add(member)
    left = np.zeros(cfg.nodes, dtype=bool)
    for _ in range(8):
        before = o.flags() >= 0
        o.step(1)
        single.step(1)
        b.step(1)
        flags = o.flags()
        left |= before & (flags < 0)
        assert np.array_equal(single.flags(), flags) and np.array_equal(member.flags(), flags)
    b.close()
    assert left.any()
