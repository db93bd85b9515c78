"""Performance cases of the RB-ThermoParticles hot path, through the public API of `rbtp`.

A user of this framework advances Rayleigh-Benard cavities: one large cavity for many steps between
two outputs, small and odd-sized ones, cavities with finite-size spheres, an ensemble of cavities in
lockstep, and restarts from stored populations.  A pass is one such stretch of work: the steps, the
Nusselt row and mean fields of its last step, and the macroscopic fields, read into page-locked
memory through the C ABI and handed to torch on the GPU, as an analysis program takes them.  Results
of the float storage modes (FP32 and shifted FP16, both with FP32 arithmetic) are kept as float32.

Inputs are a convecting state made from the seed alone on the GPU: the conduction profile with a
large-scale divergence-free roll, its temperature disturbance and a small random perturbation, as
populations at their second-order equilibrium.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "rb-thermoparticles_gb300"))
import rbtp  # noqa: E402

STORAGE = {"f64": rbtp.STORE_F64, "f32": rbtp.STORE_F32, "f16s": rbtp.STORE_F16S}
VALUE_BYTES = {"f64": 8, "f32": 4, "f16s": 2}
BETA, T_HOT, T_COLD, T_REF = 0.0000625, 1.0, 0.0, 0.5

# D3Q27 as the reference numbers it (src_lbm/initial.cu:276-286)
CX = (0, 1, 0, -1, 0, 0, 0, 1, -1, -1, 1, 1, 0, -1, 0, 1, 0, -1, 0, 1, -1, -1, 1, 1, -1, -1, 1)
CY = (0, 0, 1, 0, -1, 0, 0, 1, 1, -1, -1, 0, 1, 0, -1, 0, 1, 0, -1, 1, 1, -1, -1, 1, 1, -1, -1)
CZ = (0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, 1, 1, 1, -1, -1, -1, -1, 1, 1, 1, 1, -1, -1, -1, -1)
DIRS = list(zip(CX, CY, CZ))
OPP = [DIRS.index((-x, -y, -z)) for x, y, z in DIRS]
WEIGHT = [(8 / 27, 2 / 27, 1 / 54, 1 / 216)[abs(x) + abs(y) + abs(z)] for x, y, z in DIRS]

FLOPS_PER_NODE = 590          # of one f and g update: moments, both collisions


def _single(name, storage, lx, ly, lz, ra, steps, pr=0.71):
    return {"name": name, "kind": "steps", "storage": storage, "lx": lx, "ly": ly, "lz": lz, "ra": ra, "pr": pr,
            "steps": steps, "spheres": 0, "diameter": 0.0}


def listed():
    return [
        # the smallest cavity of the tests and of the ensembles, in the default precision, between
        # two outputs of the default cadence (125 steps): launches and latency
        _single("cavity_32_f64", "f64", 32, 32, 16, 2e4, 125),
        # the plain FP64 parity configuration, the same stretch
        _single("plain_64_f64", "f64", 64, 64, 32, 1e6, 125),
        # the same cavity in FP32, watched step by step: one step and its fields per call
        _single("plain_64_f32_watched", "f32", 64, 64, 32, 1e6, 1),
        # odd extents of a resolution study, FP64 and FP32
        _single("ragged_113_f64", "f64", 113, 87, 51, 1e6, 50),
        _single("ragged_203_f32", "f32", 203, 117, 61, 5e6, 50),
        # the production cavity (320x320x160, Ra = 1e8) in each storage mode
        _single("production_f64", "f64", 320, 320, 160, 1e8, 20),
        _single("production_f32", "f32", 320, 320, 160, 1e8, 125),
        _single("production_f16s", "f16s", 320, 320, 160, 1e8, 125),
        # parameters.h as shipped: 320x320x160, Ra = 1e7, FP64, 5 % spheres of diameter LX/20
        {"name": "default_spheres_f64", "kind": "steps", "storage": "f64", "lx": 320, "ly": 320, "lz": 160, "ra": 1e7,
         "pr": 0.71, "steps": 10, "spheres": 382, "diameter": 16.0},
        # the particle-laden production cavity: 1000 spheres of diameter 16, FP32
        {"name": "spheres_1000_f32", "kind": "steps", "storage": "f32", "lx": 320, "ly": 320, "lz": 160, "ra": 1e8,
         "pr": 0.71, "steps": 50, "spheres": 1000, "diameter": 16.0},
        # an ensemble of small cavities of mixed sizes in lockstep, half of them with spheres
        {"name": "ensemble_32_f32", "kind": "batch", "storage": "f32", "members": 32, "smallest": 32, "largest": 96,
         "ra": 1e6, "pr": 0.71, "steps": 50, "with_spheres": True},
        # a restart: FP64 populations from page-locked host memory, a few steps ending in a
        # flow-output step (dissipation fields), and the populations back for the next restart file
        {"name": "restart_160_f64", "kind": "restart", "storage": "f64", "lx": 160, "ly": 160, "lz": 80, "ra": 1e7,
         "pr": 0.71, "steps": 4},
    ]


def _stable_ra(lx, pr, want):
    """The largest Rayleigh number up to `want` whose viscosity, 0.1414 LX sqrt(Pr/Ra), stays >= 0.007
    and whose diffusivity, the viscosity over Pr, stays >= 0.0035."""
    return float(min(want, pr * (0.1414 * lx / max(0.007, 0.0035 * pr)) ** 2))


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges: extents 32..320 over their logarithm (odd ones as they
    come), 1..125 steps, each storage mode, with and without spheres, ensembles, restarts."""
    kind = rng.choice(["steps", "steps", "steps", "spheres", "spheres", "batch", "restart"])
    storage = rng.choice(["f64", "f64", "f32", "f32", "f16s"])
    pr = round(rng.uniform(0.7, 7.0), 2)
    if kind == "batch":
        lo = rng.choice([24, 32, 40, 48])
        hi = rng.choice([56, 64, 80, 96])
        return {"kind": "batch", "storage": storage, "members": rng.randint(4, 32), "smallest": lo, "largest": hi,
                "ra": round(_log(rng, 1e5, 1e6)), "pr": pr, "steps": rng.randint(5, 30),
                "with_spheres": rng.random() < 0.5}
    lx = int(_log(rng, 48 if kind == "spheres" else 32, 320))
    ly = min(320, max(24, int(lx * rng.uniform(0.6, 1.3))))
    lz = min(160, max(16 if kind != "spheres" else 32, int(lx * rng.uniform(0.3, 0.6))))
    nodes = lx * ly * lz
    case = {"kind": "steps", "storage": storage, "lx": lx, "ly": ly, "lz": lz,
            "ra": round(_stable_ra(lx, pr, _log(rng, 1e5, 1e8))), "pr": pr}
    most = (3.2e8 if storage == "f64" else 1.6e9) / (2 if kind == "spheres" else 1)
    steps = int(max(1, min(_log(rng, 1, 125), most / nodes)))
    if kind == "restart":
        return dict(case, kind="restart", lx=min(lx, 160), ly=min(ly, 160), lz=min(lz, 80), steps=min(steps, 16))
    case["steps"] = steps
    case["spheres"], case["diameter"] = 0, 0.0
    if kind == "spheres":
        d = round(rng.uniform(8.0, min(ly, lz, 80) / 4.0 + 1e-9), 3)
        case["diameter"] = d
        case["spheres"] = max(1, int(rng.uniform(0.01, 0.06) * nodes / (math.pi * d ** 3 / 6.0)))
    return case


# -------------------------------------------------------------------------------------------------
# inputs
# -------------------------------------------------------------------------------------------------
def _visc(lx, ra, pr):
    return 0.1414 * lx * math.sqrt(pr / ra)


def _config(case, seed):
    lx, ly, lz = case["lx"], case["ly"], case["lz"]
    kw = dict(lx=lx, ly=ly, lz=lz, rayleigh=float(case["ra"]), prandtl=float(case["pr"]),
              visc=_visc(lx, case["ra"], case["pr"]), storage=STORAGE[case["storage"]], activate_particles=0,
              particle_fraction=0.0, nend=1 << 30, ndiag=0, nflowout=0, nnuout=0, nout_p=0)
    if case.get("spheres"):
        volume = math.pi * case["diameter"] ** 3 / 6.0
        kw.update(activate_particles=1, particle_diam_frac=case["diameter"] / lx,
                  particle_fraction=(case["spheres"] + 0.5) * volume / (lx * ly * lz), rho_particle_ratio=1.0,
                  particle_rand_seed=86143 + int(seed) % 100000)
    return rbtp.Config.defaults(**kw)


def _state(case, seed, amplitude=0.03):
    """(f, g), float64 (27, lz, ly, lx) each, on the GPU."""
    lx, ly, lz = case["lx"], case["ly"], case["lz"]
    rng = np.random.default_rng(int(seed))
    a = amplitude * rng.uniform(0.6, 1.0, 2)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    like = dict(dtype=torch.float64, device="cuda")
    x = ((torch.arange(lx, **like) + 0.5) / lx).view(1, 1, lx)
    y = ((torch.arange(ly, **like) + 0.5) / ly).view(1, ly, 1)
    z = ((torch.arange(lz, **like) + 0.5) / lz).view(lz, 1, 1)
    pi = math.pi
    # stream function sin^2(pi x) sin^2(m pi y) sin^2(pi z): zero velocity on every wall
    m = int(rng.integers(1, 3))
    sx, sy, sz = torch.sin(pi * x) ** 2, torch.sin(m * pi * y) ** 2, torch.sin(pi * z) ** 2
    ux = a[0] * sx * torch.sin(2 * m * pi * y) * m * (lx / ly) * sz / max(1.0, m * lx / ly)
    uy = -a[0] * torch.sin(2 * pi * x) * sy * sz / max(1.0, m * lx / ly)
    uz = a[1] * 0.2 * torch.sin(pi * x) ** 2 * torch.sin(pi * y) ** 2 * torch.sin(2 * pi * z)
    t = T_HOT - x * (T_HOT - T_COLD) + 0.15 * torch.sin(pi * x) * torch.cos(m * pi * y) * torch.sin(pi * z)
    t = t + 2e-3 * (torch.rand((lz, ly, lx), generator=gen, **like) - 0.5)
    rho = 1e-4 * (torch.rand((lz, ly, lx), generator=gen, **like) - 0.5)
    f = torch.empty((27, lz, ly, lx), **like)
    g = torch.empty((27, lz, ly, lx), **like)
    u2 = ux * ux + uy * uy + uz * uz
    for i in range(27):
        cu = CX[i] * ux + CY[i] * uy + CZ[i] * uz
        e = 3.0 * cu + 4.5 * cu * cu - 1.5 * u2
        f[i] = WEIGHT[i] * (rho + e)
        g[i] = WEIGHT[i] * t * (1.0 + e)
    return f, g


def _load(solver, case, seed, amplitude=0.03):
    rows = None
    if solver.npart:
        solver.initialize()                  # the reference's seeded rejection sampling
        rows = solver.particles()
    f, g = _state(case, seed, amplitude)
    torch.cuda.synchronize()
    solver.load_state_ptr(f.data_ptr(), g.data_ptr(), None, rows)


def _member(case, k, seed):
    """Member k of an ensemble: extents spread from the smallest to the largest, LY = LX, LZ = LX/2."""
    n = case["members"]
    lx = int(round(case["smallest"] * (case["largest"] / case["smallest"]) ** (k / max(1, n - 1))))
    c = {"lx": lx, "ly": lx, "lz": max(12, lx // 2), "storage": case["storage"], "pr": case["pr"],
         "ra": _stable_ra(lx, case["pr"], case["ra"] * (1.0 + 0.1 * k)), "spheres": 0, "diameter": 0.0}
    if case["with_spheres"] and k % 2 and lx >= 48:
        c["diameter"] = 8.0
        c["spheres"] = int(0.03 * lx * lx * c["lz"] / (math.pi * 512.0 / 6.0))
    return c


class _Fields:
    """Page-locked landing place of the macroscopic fields and their copy on the GPU."""

    def __init__(self, solver):
        cfg = solver.cfg
        shape = (5, cfg.lz, cfg.ly, cfg.lx)
        self.host = torch.empty(shape, dtype=torch.float64, pin_memory=True)
        self.device = torch.empty(shape, dtype=torch.float64, device="cuda")
        dp = ctypes.POINTER(ctypes.c_double)
        self.at = [ctypes.cast(ctypes.c_void_p(self.host[k].data_ptr()), dp) for k in range(5)]

    def read(self, solver):
        status = solver.lib.rbtp_get_macros(solver.handle, *self.at, None)
        if status:
            raise rbtp.RbtpError(status, "rbtp_get_macros")
        self.device.copy_(self.host)
        return self.device


def _kept(values, storage):
    """Results in the precision that a run of this storage mode keeps."""
    if isinstance(values, torch.Tensor):
        return values if storage == "f64" else values.to(torch.float32)
    return np.asarray(values, dtype=np.float64 if storage == "f64" else np.float32)


def prepare(case, seed):
    torch.cuda.init()
    state = {"case": case}
    if case["kind"] == "batch":
        batch, solvers, fields = rbtp.Batch(STORAGE[case["storage"]]), [], []
        for k in range(case["members"]):
            c = _member(case, k, seed)
            s = rbtp.Solver(_config(c, seed + k))
            _load(s, c, seed * 1000 + k, 0.02)
            batch.add(s, sample_every=case["steps"])
            solvers.append(s)
            fields.append(_Fields(s))
        # a serving loop's tuned choice outlives membership changes: the launch shapes are chosen here
        # (the first 16 steps), in whole stretches so that every pass ends on a sampled step
        batch.step(case["steps"] * -(-16 // case["steps"]))
        for s in solvers:
            batch.samples(s)
        state.update(batch=batch, solvers=solvers, fields=fields)
    elif case["kind"] == "restart":
        s = rbtp.Solver(_config(case, seed))
        dp = ctypes.POINTER(ctypes.c_double)
        shape = (2, 27, case["lz"], case["ly"], case["lx"])
        src, back = (torch.empty(shape, dtype=torch.float64, pin_memory=True) for _ in range(2))
        f, g = _state(case, seed)
        src[0].copy_(f)
        src[1].copy_(g)
        del f, g
        diss = torch.empty((2,) + shape[2:], dtype=torch.float64, pin_memory=True)
        at = [ctypes.cast(ctypes.c_void_p(t.data_ptr()), dp) for t in (back[0], back[1], diss[0], diss[1])]
        state.update(solver=s, src=src, back=back, diss=diss, at=at, fields=_Fields(s))
    else:
        s = rbtp.Solver(_config(case, seed))
        _load(s, case, seed)
        state.update(solver=s, fields=_Fields(s))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return state


def run(state):
    case = state["case"]
    storage = case["storage"]
    if case["kind"] == "batch":
        state["batch"].step(case["steps"])
        nu = [state["batch"].samples(s)[-1][1:] for s in state["solvers"]]
        out = {"nu": _kept(np.stack(nu), storage),
               "fields": [_kept(fl.read(s), storage) for s, fl in zip(state["solvers"], state["fields"])]}
        rows = [s.particles() for s in state["solvers"] if s.npart]
        if rows:
            out["spheres"] = _kept(np.concatenate(rows), storage)
        return out
    s = state["solver"]
    if case["kind"] == "restart":
        s.load_state_ptr(state["src"][0].data_ptr(), state["src"][1].data_ptr())
        s.step(case["steps"], macros_last=True, flow_last=True)
        f_at, g_at, ted_at, ked_at = state["at"]
        for status in (s.lib.rbtp_get_fg(s.handle, f_at, g_at), s.lib.rbtp_dissipation(s.handle, ted_at, ked_at)):
            if status:
                raise rbtp.RbtpError(status, "restart output")
        return {"f": _kept(state["back"][0], storage), "g": _kept(state["back"][1], storage),
                "dissipation": _kept(state["diss"], storage), "fields": _kept(state["fields"].read(s), storage)}
    s.step(case["steps"], macros_last=True)
    out = {"nu": _kept(s.nu(0)[1:], storage), "means": _kept(s.means(), storage),
           "fields": _kept(state["fields"].read(s), storage)}
    if s.npart:
        out["spheres"] = _kept(s.particles(), storage)
    return out


def work(case):
    """Every step reads and writes the 27 + 27 populations and the buoyancy of each node once; the
    fields (and for a restart the stored populations) leave or enter the GPU once."""
    v = VALUE_BYTES[case["storage"]]
    per_node = 2 * 54 * v + 2 * max(4, v)
    if case["kind"] == "batch":
        members = [_member(case, k, 0) for k in range(case["members"])]
        nodes = sum(c["lx"] * c["ly"] * c["lz"] for c in members)
    else:
        nodes = case["lx"] * case["ly"] * case["lz"]
    extra = 5 * 8 * nodes
    if case["kind"] == "restart":
        extra += (2 * 54 + 2) * 8 * nodes
    return {"bytes": float(case["steps"] * nodes * per_node + extra),
            "flops": float(case["steps"] * nodes * FLOPS_PER_NODE)}


# -------------------------------------------------------------------------------------------------
# the same step in plain torch, 64 bits
# -------------------------------------------------------------------------------------------------
class _Plain:
    """The reference's step (src_lbm/macrovar.cu, collision.cu, streaming.cu), literally."""

    def __init__(self, case, f, g):
        self.case, self.f, self.g = case, f, g
        lx, visc = case["lx"], _visc(case["lx"], case["ra"], case["pr"])
        self.grav = case["ra"] * visc * visc / (BETA * (T_HOT - T_COLD) * float(lx) ** 3 * case["pr"])
        self.tau, self.tauc = 3.0 * visc + 0.5, 3.0 * visc / case["pr"] + 0.5
        self.fx = self.grav * BETA * (g.sum(0) - T_REF)

    def _stream(self, p, rho=None):
        lz, ly, lx = p.shape[1:]
        out = torch.empty_like(p)
        for i, (cx, cy, cz) in enumerate(DIRS):
            out[i] = p[OPP[i]]
            to = tuple(slice(max(0, c), n + min(0, c)) for c, n in ((cz, lz), (cy, ly), (cx, lx)))
            at = tuple(slice(max(0, -c), n + min(0, -c)) for c, n in ((cz, lz), (cy, ly), (cx, lx)))
            out[(i,) + to] = p[(i,) + at]
            if rho is not None and cx:
                wall = (to[0], to[1], 0 if cx > 0 else lx - 1)
                t = T_HOT if cx > 0 else T_COLD
                out[(i,) + wall] = -p[(OPP[i],) + wall] + 2.0 * WEIGHT[i] * t * (1.0 + rho[wall])
        return out

    def step(self):
        f, g, tau, tauc = self.f, self.g, self.tau, self.tauc
        rho, phi = torch.zeros_like(f[0]), torch.zeros_like(f[0])
        j = [torch.zeros_like(f[0]) for _ in range(3)]
        for i, c in enumerate(DIRS):
            rho += f[i]
            phi += g[i]
            for a in range(3):
                if c[a]:
                    j[a] += c[a] * f[i]
        ux, uy, uz = j[0] + 0.5 * self.fx, j[1], j[2]
        self.fields = (rho, ux, uy, uz, phi)
        fx = self.fx = self.grav * BETA * (phi - T_REF)
        uv = 3.0 * (ux * ux + uy * uy + uz * uz)

        def terms(i):
            eu = 3.0 * (CX[i] * ux + CY[i] * uy + CZ[i] * uz)
            return eu, 0.5 * (eu * eu - uv)

        def geqnew(i):
            eu, q = terms(i)
            geq = WEIGHT[i] * phi * (1.0 + eu + q)
            return geq - (1.0 - WEIGHT[0]) * phi * rho if i == 0 else geq + WEIGHT[i] * phi * rho

        k = [torch.zeros_like(rho) for _ in range(3)]
        for i, c in enumerate(DIRS):
            d = g[i] - geqnew(i)
            for a in range(3):
                if c[a]:
                    k[a] += c[a] * d
        denom = rho / 3.0 + 2.0 * tauc / 3.0
        fc, gc = torch.empty_like(f), torch.empty_like(g)
        for i, c in enumerate(DIRS):
            eu, q = terms(i)
            feq = WEIGHT[i] * (rho + eu + q)
            feq1 = WEIGHT[i] * (1.0 + eu + q)
            fc[i] = f[i] - (f[i] - feq) / tau + (1.0 - 0.5 / tau) * 3.0 * (c[0] - ux) * fx * feq1
            eb = c[0] * fx
            gneq = c[0] * k[0] + c[1] * k[1] + c[2] * k[2]
            grad = -(2.0 * gneq + eb * phi) / denom
            src = WEIGHT[i] * (1.0 - 0.5 / tauc) * (grad * rho + 3.0 * phi * eb)
            gc[i] = g[i] - (g[i] - geqnew(i)) / tauc + src
        self.f, self.g = self._stream(fc), self._stream(gc, rho)


def exact(case, seed):
    """Single-phase passes; the coupling of moving spheres has no short plain form (None), nor have
    the restart's dissipation fields and the Nusselt row's on-device sums."""
    if case["kind"] == "batch" or case.get("spheres") or case["steps"] * case["lx"] * case["ly"] * case["lz"] > 2.2e9:
        return None
    plain = _Plain(case, *_state(case, seed))
    for _ in range(case["steps"]):
        plain.step()
    fields = torch.stack(plain.fields)
    if case["kind"] == "restart":
        return {"f": plain.f, "g": plain.g, "dissipation": None, "fields": fields}
    return {"nu": None, "means": fields[1:].mean(dim=(1, 2, 3)), "fields": fields}
