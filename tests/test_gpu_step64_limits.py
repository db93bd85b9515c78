"""The FP64 step on values that its integer grids do not take."""
import numpy as np
import pytest

from rbtp import RbtpError, Solver, workloads as W

pytestmark = pytest.mark.gpu
LX, LY, LZ = 34, 5, 4
MIDDLE, WALL = 2 * LX * LY + 2 * LX + 17, LX * LY + 2 * LX   # an inner node and one at the hot wall


def _populations(cfg, seed):
    """f, g near equilibrium of random velocities and temperatures."""
    rng = np.random.default_rng(seed)
    L = cfg.nodes
    u = 0.1 * rng.uniform(-1, 1, (3, L))
    rho, t = 1e-3 * rng.uniform(-1, 1, L), rng.uniform(0.1, 1, L)
    cu = W.CX[:, None] * u[0] + W.CY[:, None] * u[1] + W.CZ[:, None] * u[2]
    e = 3 * cu + 4.5 * cu * cu - 1.5 * (u * u).sum(0)
    return W.W[:, None] * (rho + e), W.W[:, None] * t * (1 + e)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e200])
@pytest.mark.parametrize("which,direction", [(0, 0), (0, 1), (0, 20), (1, 0), (1, 5)])
@pytest.mark.parametrize("node", [MIDDLE, WALL])
def test_a_non_finite_population_reaches_the_populations_that_it_reaches_in_plain_fp64(
        lib_built, oracle_mod, which, direction, value, node):
    cfg = W.config("plain_fp64", lx=LX, ly=LY, lz=LZ)
    fg = _populations(cfg, 1)
    fg[which][direction, node] = value
    s, o = Solver(cfg), oracle_mod.Oracle(cfg)
    for x in (s, o):
        x.load_state(fg[0].reshape(-1), fg[1].reshape(-1), None)
    for _ in range(3):
        with pytest.raises(RbtpError) as e:
            s.step(1)
        assert e.value.status == -4
        o.step(1)
        for a, b in zip(s.fg(), o.fg()):
            assert np.array_equal(np.isfinite(a), np.isfinite(b))


def _around(a, r):
    """The largest |a| over the nodes within r of each node, and over the directions."""
    m = np.abs(a).max(0).reshape(LZ, LY, LX)
    for axis in range(3):
        pad = np.pad(m, [(r, r) if k == axis else (0, 0) for k in range(3)])
        m = np.max([np.take(pad, range(d, d + m.shape[axis]), axis) for d in range(2 * r + 1)], 0)
    return m.reshape(-1)


@pytest.mark.parametrize("rho", [-0.9, -0.3, -1e-8, 1e-300, 1e-8, 0.7, 40.0, 3e4])
@pytest.mark.parametrize("prandtl", [0.02, 0.71, 50.0])
def test_density_over_the_denominator_of_the_scalar_source(lib_built, oracle_mod, rho, prandtl):
    """rho / (rho / 3 + 2 tauc / 3) of the g source, for densities and diffusivities far from any flow's.  The
    source's terms are a few times the node's largest g, and its rounding and the sums' are some ten
    of 2^-53 each: 5e-15 of the largest around."""
    cfg = W.config("plain_fp64", lx=LX, ly=LY, lz=LZ, prandtl=prandtl, visc=0.02)
    f, g = _populations(cfg, 5)
    f += W.W[:, None] * rho * np.random.default_rng(6).uniform(0.5, 1, cfg.nodes)
    s, o = Solver(cfg), oracle_mod.Oracle(cfg)
    for x in (s, o):
        x.load_state(f.reshape(-1), g.reshape(-1), None)
        x.step(1)
    for a, b in zip(s.fg(), o.fg()):
        a, b = a.reshape(27, -1), b.reshape(27, -1)
        assert np.all(np.abs(a - b) <= 5e-15 * _around(b, 1))


# Populations from 2^16 on, and coefficients of that size, take the plain FP64 path, f and g each by itself.
# "pair": the value at +x and at -x of one node, so that its velocity stays small and its coefficients below
# the limit.  "single": at +x alone; the coefficient 9 u^2 / (216 tau) reaches 2^16 near u = 1.2e3.
@pytest.mark.parametrize("node", [MIDDLE, WALL])
@pytest.mark.parametrize("kind,which,value", [
    ("pair", w, v) for w in (0, 1) for v in (2.0 ** 15, np.nextafter(2.0 ** 16, 0), 2.0 ** 16, 2.0 ** 17, 2.0 ** 19)] + [
    ("single", 0, v) for v in (90.0, 1100.0, 1300.0, 2.0 ** 15)] + [
    ("single", 1, v) for v in (2.0 ** 15, np.nextafter(2.0 ** 16, 0), 2.0 ** 16, 2.0 ** 17)])
def test_both_sides_of_the_grids_limit_node_by_node(lib_built, oracle_mod, kind, which, value, node):
    """A node's populations carry some ten roundings of 2^-53 of the largest term of the node they come from, so the
    first (even) step lies within 5e-15 of the largest |f| around; the second (odd) one doubles the relative error
    of u in u^2 and meets the first one's in k1: 4 times that.  Nodes out of reach of the value are compared with
    what is around them alone, so they may not notice it."""
    cfg = W.config("plain_fp64", lx=LX, ly=LY, lz=LZ)
    fg = _populations(cfg, 8)
    for d in (1, 3) if kind == "pair" else (1,):
        fg[which][d, node] = value
    s, o = Solver(cfg), oracle_mod.Oracle(cfg)
    for x in (s, o):
        x.load_state(fg[0].reshape(-1), fg[1].reshape(-1), None)
    for step in (1, 2):
        s.step(1, macros_last=True)
        o.step(1)
        for a, b in zip(s.fg(), o.fg()):
            a, b = a.reshape(27, -1), b.reshape(27, -1)
            assert np.all(np.abs(a - b) <= 5e-15 * 4 ** (step - 1) * _around(b, 1))
