"""The FP64 step's integer-unit sums at the edges of their ranges: row remainders of the 32-node warps,
populations 2^-300 to 1 times their size within a node, values far beyond the grids' limit of 2^16 (the
plain FP64 path), and non-finite ones.  Against the oracle's plain FP64 formulas; the tolerance is a few roundings (2^-53
each) of the node's largest terms per step, over at most four steps."""
import numpy as np
import pytest

from conftest import rel_l2
from rbtp import Batch, RbtpError, Solver, workloads as W

pytestmark = pytest.mark.gpu
TOL = 5e-15


def _pair(oracle_mod, lx, ly, lz, f, g):
    cfg = W.config("plain_fp64", lx=lx, ly=ly, lz=lz)
    s, o = Solver(cfg), oracle_mod.Oracle(cfg)
    s.load_state(f, g, None)
    o.load_state(f, g, None)
    return s, o


def _populations(lx, ly, lz, seed, spread):
    """f, g near equilibrium of random velocities; `spread` scales each population by 2^-U(0, spread)."""
    rng = np.random.default_rng(seed)
    L = lx * ly * lz
    u = 0.1 * rng.uniform(-1, 1, (3, L))
    rho, t = 1e-3 * rng.uniform(-1, 1, L), rng.uniform(0, 1, L)
    cu = W.CX[:, None] * u[0] + W.CY[:, None] * u[1] + W.CZ[:, None] * u[2]
    e = 3 * cu + 4.5 * cu * cu - 1.5 * (u * u).sum(0)
    scale = np.exp2(-rng.uniform(0, spread, (27, L))) if spread else 1.0
    return (scale * W.W[:, None] * (rho + e)).reshape(-1), (scale * W.W[:, None] * t * (1 + e)).reshape(-1)


def _close(s, o, tol=TOL):
    for a, b in zip(s.fg(), o.fg()):
        assert rel_l2(a, b) < tol, rel_l2(a, b)
    ms, mo = s.macros(), o.macros()
    for k in ("rho", "ux", "uy", "uz", "phi", "force_x"):
        assert np.linalg.norm(ms[k] - mo[k]) <= tol * max(np.linalg.norm(mo[k]), 1e-2 * np.linalg.norm(mo["phi"])), k


@pytest.mark.parametrize("lx,ly,lz", [(3, 3, 3), (31, 5, 4), (32, 3, 5), (33, 4, 3), (65, 7, 3)])
@pytest.mark.parametrize("spread", [0, 30, 300])
def test_sizes_and_exponents(lib_built, oracle_mod, lx, ly, lz, spread):
    s, o = _pair(oracle_mod, lx, ly, lz, *_populations(lx, ly, lz, lx + spread, spread))
    for _ in range(4):
        s.step(1, macros_last=True)
        o.step(1)
        _close(s, o)


def test_zero_and_mirrored_states_stay_exact(lib_built, oracle_mod):
    L = 40 * 6 * 5
    g = (W.W[:, None] * np.full(L, 0.5)).reshape(-1)
    s, o = _pair(oracle_mod, 40, 6, 5, np.zeros(27 * L), np.zeros(27 * L))
    s.step(1, macros_last=True)
    o.step(1)
    assert np.all(s.macros()["rho"] == 0) and np.all(s.macros()["uy"] == 0)
    s, o = _pair(oracle_mod, 40, 6, 5, np.zeros(27 * L), g)
    s.step(2, macros_last=True)
    # the arithmetic is odd: the mirrored half is the exact negative
    for k, axis in (("uy", 1), ("uz", 0)):
        u = s.macros()[k].reshape(5, 6, 40)
        assert np.array_equal(u, -np.flip(u, axis)), k


@pytest.mark.parametrize("value", [2.0 ** 89, 2.0 ** 90, 1e28])
def test_values_at_and_beyond_the_grids(lib_built, oracle_mod, value):
    lx, ly, lz = 34, 5, 4
    f, g = _populations(lx, ly, lz, 7, 0)
    L = lx * ly * lz
    f[3 * L + 100] = value          # one population of one node in the middle
    f[9 * L] = -value               # and one at a corner of the box
    s, o = _pair(oracle_mod, lx, ly, lz, f, g)
    s.step(1, macros_last=True)
    o.step(1)
    _close(s, o, 1e-14)


@pytest.mark.parametrize("which,value", [(0, np.nan), (1, np.inf), (1, np.nan), (0, 1e31)])
def test_non_finite_values_are_reported(lib_built, which, value):
    cfg = W.config("plain_fp64", lx=33, ly=5, lz=4)
    fg = list(_populations(33, 5, 4, 3, 0))
    fg[which][5 * cfg.nodes + 50] = value
    s = Solver(cfg)
    s.load_state(*fg, None)
    with pytest.raises(RbtpError) as e:
        s.step(1)
    assert e.value.status == -4


def test_batched_fp64_members_of_ragged_sizes_match_single_runs(lib_built):
    sizes = [(3, 3, 3), (33, 5, 6), (64, 3, 4), (65, 9, 5)]
    runs = []
    for batched in (False, True):
        solvers = []
        for k, (lx, ly, lz) in enumerate(sizes):
            s = Solver(W.config("plain_fp64", lx=lx, ly=ly, lz=lz))
            s.load_state(*_populations(lx, ly, lz, k, 5), None)
            solvers.append(s)
        if batched:
            b = Batch(0)
            for s in solvers:
                b.add(s)
            b.step(21)
        else:
            for s in solvers:
                s.step(21)
        runs.append([s.fg() for s in solvers])
        if batched:
            b.close()
    for x, y in zip(*runs):
        assert np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1])


# 64 x 57 nodes are 114 blocks of a plane: 12 and 16 planes take each choice of resident blocks, 48 are
# the last that the unrolled step takes
@pytest.mark.parametrize("lz", [12, 16, 48, 49])
def test_all_variants_give_the_same_bits(lib_built, lz):
    fg = _populations(64, 57, lz, lz, 5)
    runs = []
    for batched in (False, True):
        s = Solver(W.config("plain_fp64", lx=64, ly=57, lz=lz))
        s.load_state(*fg, None)
        if batched:
            b = Batch(0)
            b.add(s)
            b.step(3)
            b.close()
        else:
            s.step(3)
        runs.append(s.fg())
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
