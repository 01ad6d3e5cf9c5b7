"""The workloads whose speed is followed: molecular-dynamics runs, observables and training
steps as a program that uses this package has it do, through the C ABI that the package's
classes call (include/espp_b200.h), with the layout the library chooses by itself.

The sizes are those of the benchmark configurations (32,768 and 4,096,000 particle
Lennard-Jones fluids, the 40,000-bead Kremer-Grest melt, parallel-tempering replicas of a
few thousand particles, 50,000 coarse-grained sites) with the 2,000-particle fluid of the
tests below them and ragged boxes between.

Every start configuration comes from the seed alone: particles on a jittered lattice with
Maxwell-Boltzmann velocities.  A pass continues the run from where the last one ended.
"""
import ctypes
import math

import numpy as np
import torch

from espressopp_b200 import _abi, load_library
from espressopp_b200._abi import call, dptr, i32ptr, i64ptr

RHO = 0.8442          # fluid density of the benchmark configurations
RC, SKIN = 2.5, 0.3
RC_WCA = 2.0 ** (1.0 / 6.0)
RHO_MELT = 0.85
RHO_CG = 0.85 / 4.0   # sites of 4 beads
RC_CG, R0_CG = 3.0, 0.5
RDF_BINS = 256
MLP_K, MLP_H = 16, 64


# ---- the cases -----------------------------------------------------------------------
def listed():
    return [
        # the smallest runs a user does (the tests' 2048-particle fluid): launches and
        # host work count; few steps a call, as when observables are sampled often
        {"name": "fluid_2k_fp64", "kind": "fluid", "nx": 13, "ny": 13, "nz": 12,
         "precision": "fp64", "langevin": True, "types": 1, "steps": 20},
        # the thermostatted 32,768-particle fluid in both precisions
        {"name": "fluid_32k_fp64", "kind": "fluid", "nx": 32, "ny": 32, "nz": 32,
         "precision": "fp64", "langevin": True, "types": 1, "steps": 100},
        {"name": "fluid_32k_mixed", "kind": "fluid", "nx": 32, "ny": 32, "nz": 32,
         "precision": "mixed", "langevin": True, "types": 1, "steps": 100},
        # a binary mixture in a box of unequal edges: per-pair parameters, ragged sizes
        {"name": "mixture_241k_mixed", "kind": "fluid", "nx": 61, "ny": 67, "nz": 59,
         "precision": "mixed", "langevin": True, "types": 2, "steps": 50},
        # a large NVE fluid in reference arithmetic, the default precision
        {"name": "fluid_1m_fp64", "kind": "fluid", "nx": 97, "ny": 101, "nz": 103,
         "precision": "fp64", "langevin": False, "types": 1, "steps": 40},
        # the benchmark's headline fluid
        {"name": "fluid_4m_mixed", "kind": "fluid", "nx": 160, "ny": 160, "nz": 160,
         "precision": "mixed", "langevin": False, "types": 1, "steps": 40},
        # the Kremer-Grest melt: short cutoff, FENE bonds
        {"name": "melt_40k_mixed", "kind": "melt", "nx": 40, "ny": 40, "nz": 25,
         "beads": 200, "precision": "mixed", "steps": 50},
        # parallel-tempering replicas of uneven size between two exchanges
        {"name": "replicas_24", "kind": "replicas", "count": 24, "smin": 13, "smax": 25,
         "precision": "mixed", "steps": 50},
        # structure of a configuration: every pair of particles
        {"name": "rdf_32k", "kind": "rdf", "nx": 32, "ny": 32, "nz": 32},
        # energy and pressure tensor of a large configuration
        {"name": "observables_1m", "kind": "observables", "nx": 97, "ny": 101, "nz": 103},
        # one training step of the learned potential on one frame (BF16 network)
        {"name": "train_50k", "kind": "train", "nx": 37, "ny": 37, "nz": 37},
        # a coarse-grained run: bond, angle and pair tables with the learned potential
        {"name": "cg_50k", "kind": "cg", "nx": 50, "ny": 40, "nz": 25, "beads": 50,
         "steps": 30},
    ]


def _sides(rng, n, least):
    """Three lattice edges whose product is about n, not all equal as a rule."""
    a = n ** (1.0 / 3.0)
    nx = max(least, int(round(a * rng.uniform(0.85, 1.18))))
    ny = max(least, int(round(a * rng.uniform(0.9, 1.1))))
    return nx, ny, max(least, int(round(n / (nx * ny))))


def draw(rng):
    kind = rng.choice(["fluid"] * 5 + ["melt"] * 2 + ["replicas", "rdf", "observables",
                                                      "train", "cg"])
    spread = lambda lo, hi: math.exp(rng.uniform(math.log(lo), math.log(hi)))  # noqa: E731
    if kind == "fluid":
        n = spread(2.1e3, 3.6e6)
        nx, ny, nz = _sides(rng, n, 11)
        top = 100 if n < 3e5 else 20
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz,
                "precision": rng.choice(["fp64", "mixed"]) if n < 1.1e6 else "mixed",
                "langevin": rng.random() < 0.5, "types": rng.choice([1, 1, 2]),
                "steps": rng.randint(5, top)}
    if kind == "melt":
        nx, ny, nz = _sides(rng, spread(4e3, 2e5), 11)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "beads": rng.choice([50, 100, 200]),
                "precision": rng.choice(["fp64", "mixed"]), "steps": rng.randint(10, 50)}
    if kind == "replicas":
        return {"kind": kind, "count": rng.randint(4, 24), "smin": 13,
                "smax": rng.randint(15, 25), "precision": rng.choice(["fp64", "mixed"]),
                "steps": rng.randint(10, 50)}
    if kind == "rdf":
        nx, ny, nz = _sides(rng, spread(2.1e3, 3.2e4), 11)
    elif kind == "observables":
        nx, ny, nz = _sides(rng, spread(2.1e3, 1.0e6), 11)
    else:
        nx, ny, nz = _sides(rng, spread(6e3, 5e4), 10)
    case = {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    if kind == "cg":
        case.update(beads=rng.choice([25, 50]), steps=rng.randint(5, 30))
    return case


# ---- configurations --------------------------------------------------------------------
def _lattice(nx, ny, nz, rho, jitter, g):
    """Sites (n, 3) of a simple cubic lattice, x fastest, each moved by up to +-jitter."""
    a = rho ** (-1.0 / 3.0)
    n = nx * ny * nz
    k = np.arange(n)
    pos = np.empty((n, 3))
    pos[:, 0], pos[:, 1], pos[:, 2] = k % nx, (k // nx) % ny, k // (nx * ny)
    pos = (pos + 0.5) * a + g.uniform(-jitter, jitter, (n, 3))
    return pos, np.array([nx * a, ny * a, nz * a])


def _chain_lattice(nx, ny, nz, rho, jitter, g):
    """The same lattice in the order of a walk that visits every site once, each step to a
    neighbouring site: a dense melt of straight and folded chain pieces."""
    pos, box = _lattice(nx, ny, nz, rho, jitter, g)
    site = np.arange(nx * ny * nz).reshape(nz, ny, nx).copy()
    site[1::2] = site[1::2, ::-1]       # every second layer is walked row by row backwards
    rows = site.reshape(nz * ny, nx)
    rows[1::2] = rows[1::2, ::-1]       # every second row is walked backwards
    return pos[rows.reshape(-1)], box


def _velocities(n, T, g):
    v = g.normal(0.0, math.sqrt(T), (n, 3))
    return v - v.mean(0)


def _bonds(n, beads):
    k = np.arange(n - 1, dtype=np.int64)
    k = k[(k + 1) % beads != 0]
    return np.stack([k, k + 1], 1)


def _triples(n, beads):
    k = np.arange(n - 2, dtype=np.int64)
    k = k[((k + 1) % beads != 0) & ((k + 2) % beads != 0)]
    return np.stack([k, k + 1, k + 2], 1)


# LJ parameters (epsilon, sigma) by type pair: one type, or the 80:20 mixture of Kob and
# Andersen, each truncated at 2.5 sigma
_LJ = {1: {(0, 0): (1.0, 1.0)},
       2: {(0, 0): (1.0, 1.0), (0, 1): (1.5, 0.8), (1, 1): (0.5, 0.88)}}


def _lj_terms(case):
    if case["kind"] == "melt":
        return {(0, 0): (1.0, 1.0, RC_WCA)}
    return {k: (e, s, RC * s) for k, (e, s) in _LJ[case.get("types", 1)].items()}


def _particles(case, seed):
    """(pos, vel, types, box) of a case; masses are 1 (4 for coarse-grained sites)."""
    g = np.random.Generator(np.random.PCG64(seed))
    kind = case["kind"]
    shape = (case["nx"], case["ny"], case["nz"])
    if kind == "melt":
        pos, box = _chain_lattice(*shape, RHO_MELT, 0.05, g)
    elif kind == "cg":
        pos, box = _chain_lattice(*shape, RHO_CG, 0.15, g)
    elif kind == "train":
        pos, box = _lattice(*shape, RHO_CG, 0.3, g)
    else:
        pos, box = _lattice(*shape, RHO, 0.05, g)
    n = len(pos)
    vel = _velocities(n, 0.25 if kind == "cg" else 1.0, g)
    typ = (g.random(n) < 0.2).astype(np.int32) if case.get("types", 1) == 2 else np.zeros(n, np.int32)
    return pos, vel, typ, box, g


def _mlp_params(g):
    K, H = MLP_K, MLP_H
    return np.concatenate([g.normal(0, 1 / math.sqrt(K), H * K), g.normal(0, 0.1, H),
                           g.normal(0, 1 / math.sqrt(H), H * H), g.normal(0, 0.1, H),
                           g.normal(0, 0.1 / math.sqrt(H), H), [0.0]])


def _mlp_norm():
    """Mean and inverse spread of the descriptors of a uniform fluid of sites."""
    r = np.linspace(1e-3, RC_CG, 4000)
    w = (RC_CG - R0_CG) / (MLP_K - 1)
    mu = R0_CG + w * np.arange(MLP_K)
    gk = np.exp(-(r[:, None] - mu) ** 2 / (2 * w * w)) * ((np.cos(np.pi * r / RC_CG) + 1) / 2)[:, None]
    shell = (4 * np.pi * RHO_CG * r * r * (r[1] - r[0]) * (r > 1.0))[:, None]
    sd = np.sqrt((shell * gk * gk).sum(0))
    return (shell * gk).sum(0), 1.0 / np.sqrt(sd * sd + (0.1 * sd.max()) ** 2)


# tables of the coarse-grained run: harmonic-like bonds about the lattice spacing, a weak
# stiffness of the angles, a soft repulsion between sites
def _bond_table():
    r = np.linspace(0.05, 8.0, 400)
    return r, 10.0 * (r - 1.68) ** 2, -20.0 * (r - 1.68)


def _angle_table():
    t = np.linspace(0.0, math.pi, 721)
    return t, 2.0 * (1.0 + np.cos(t)), 2.0 * np.sin(t)


def _pair_table():
    r = np.linspace(0.05, RC_CG, 400)
    x = np.clip(1.0 - r / RC_CG, 0.0, None)
    return r, 6.0 * x ** 3, 18.0 * x ** 2 / RC_CG


class _Sys:
    """One system of the library with the buffers its results are read into."""

    def __init__(self, box, rc, skin, precision, seed):
        self.lib = load_library()
        self.h = ctypes.c_void_p()
        self.box = np.ascontiguousarray(box, np.float64)
        cg = np.array([max(3, int(b / (rc + skin))) for b in box], np.int32)
        prec = _abi.PREC_FP64 if precision == "fp64" else _abi.PREC_MIXED
        call(self.lib, "espp_system_create", dptr(self.box), skin, i32ptr(cg), prec, seed,
             ctypes.byref(self.h))
        self.model = None

    def add(self, pos, vel, typ=None, mass=None):
        self.n = len(pos)
        self.ids = np.arange(self.n, dtype=np.int64)
        call(self.lib, "espp_add_particles", self.h, self.n, i64ptr(self.ids),
             None if typ is None else i32ptr(typ), dptr(mass), dptr(np.ascontiguousarray(pos)),
             dptr(np.ascontiguousarray(vel)))
        call(self.lib, "espp_decompose", self.h)

    def lj(self, terms):
        for (a, b), (eps, sig, rc) in terms.items():
            q = (sig / rc) ** 6
            call(self.lib, "espp_lj_set", self.h, a, b, eps, sig, rc, 4.0 * eps * (q * q - q), 0.0)

    def run(self, steps):
        call(self.lib, "espp_run", self.h, steps)

    def read(self, out):
        call(self.lib, "espp_get_particles", self.h, self.n, i64ptr(self.ids), dptr(out[0]),
             dptr(out[1]), dptr(out[2]), None)

    def __del__(self):
        try:
            if self.h:
                self.lib.espp_system_destroy(self.h)
            if self.model:
                self.lib.espp_mlp_destroy(self.model)
        except Exception:
            pass


def _pinned(*shape):
    t = torch.empty(shape, dtype=torch.float64)
    return t.pin_memory() if torch.cuda.is_available() else t


def _make(case, seed):
    pos, vel, typ, box, g = _particles(case, seed)
    kind = case["kind"]
    rc = {"melt": RC_WCA, "cg": RC_CG, "train": RC_CG}.get(kind, RC)
    s = _Sys(box, rc, SKIN, case.get("precision", "mixed" if kind in ("cg", "train") else "fp64"),
             seed + 1)
    mass = np.full(len(pos), 4.0) if kind in ("cg", "train") else None
    s.add(pos, vel, typ, mass)
    call(s.lib, "espp_vl_create", s.h, rc, 0, None)
    if kind in ("cg", "train"):
        s.model = ctypes.c_void_p()
        call(s.lib, "espp_mlp_create", RC_CG, R0_CG, ctypes.byref(s.model))
        theta = np.ascontiguousarray(_mlp_params(g))
        call(s.lib, "espp_mlp_set_params", s.model, len(theta), dptr(theta))
        shift, scale = (np.ascontiguousarray(a) for a in _mlp_norm())
        call(s.lib, "espp_mlp_set_norm", s.model, dptr(shift), dptr(scale))
        call(s.lib, "espp_mlp_attach", s.h, s.model)
    if kind == "cg":
        b = _bonds(s.n, case["beads"])
        t = _triples(s.n, case["beads"])
        call(s.lib, "espp_bonds_add", s.h, len(b), i64ptr(b))
        call(s.lib, "espp_triples_add", s.h, len(t), i64ptr(t))
        for name, tab, tail in (("espp_tab_bond_set", _bond_table(), (math.inf, 0.0)),
                                ("espp_tab_angle_set", _angle_table(), ())):
            r, e, f = (np.ascontiguousarray(a) for a in tab)
            call(s.lib, name, s.h, _abi.TAB_LINEAR, len(r), dptr(r), dptr(e), dptr(f), *tail)
        r, e, f = (np.ascontiguousarray(a) for a in _pair_table())
        call(s.lib, "espp_tab_pair_set", s.h, 0, 0, _abi.TAB_LINEAR, len(r), dptr(r), dptr(e),
             dptr(f), RC_CG, 0.0)
    elif kind != "train":
        s.lj(_lj_terms(case))
    if kind == "melt":
        b = _bonds(s.n, case["beads"])
        call(s.lib, "espp_bonds_add", s.h, len(b), i64ptr(b))
        call(s.lib, "espp_fene_set", s.h, 30.0, 0.0, 1.5, math.inf, 0.0)
    dt, lang = _dynamics(case)
    call(s.lib, "espp_integrator_set", s.h, dt)
    if lang:
        call(s.lib, "espp_langevin_set", s.h, 1, lang[0], lang[1], 0, None)
    if kind == "train":
        s.frame = np.ascontiguousarray(pos - box * np.floor(pos / box))
        s.target = np.ascontiguousarray(g.normal(0.0, 3.0, (s.n, 3)))
        s.grad = np.empty(len(theta))
        s.theta = np.empty(len(theta))
    return s


def _dynamics(case):
    """(dt, (gamma, T) of the thermostat or None)."""
    if case["kind"] in ("melt", "cg"):
        return 0.01, (0.5, 1.0)
    return 0.005, (1.0, case.get("temperature", 1.0)) if case.get("langevin") else None


def _replica_cases(case):
    """The replicas: cubic fluids of uneven size, temperatures geometric from 0.7 to 2."""
    g = np.random.Generator(np.random.PCG64([case["count"], case["smin"], case["smax"]]))
    R = case["count"]
    out = []
    for r in range(R):
        n = int(g.integers(case["smin"], case["smax"] + 1))
        out.append({"kind": "fluid", "nx": n, "ny": n, "nz": n, "precision": case["precision"],
                    "langevin": True, "types": 1, "steps": case["steps"],
                    "temperature": 0.7 * (2.0 / 0.7) ** (r / max(R - 1, 1))})
    return out


class _Replicas:
    def __init__(self, case, seed):
        self.sys = [_make(c, seed + 1000 * (k + 1))
                    for k, c in enumerate(_replica_cases(case))]
        self.lib = self.sys[0].lib
        arr = (ctypes.c_void_p * len(self.sys))(*[s.h.value for s in self.sys])
        self.b = ctypes.c_void_p()
        call(self.lib, "espp_batch_create", arr, len(self.sys), ctypes.byref(self.b))
        total = sum(s.n for s in self.sys)
        self.out = [_pinned(total, 3) for _ in range(3)]
        self.rows = []
        at = 0
        for s in self.sys:
            self.rows.append([o[at:at + s.n].numpy() for o in self.out])
            at += s.n

    def __del__(self):
        try:
            self.lib.espp_batch_destroy(self.b)
        except Exception:
            pass


def prepare(case, seed):
    kind = case["kind"]
    if kind == "replicas":
        return case, _Replicas(case, seed)
    s = _make(case, seed)
    if kind in ("fluid", "melt", "cg"):
        s.out = [_pinned(s.n, 3) for _ in range(3)]
        s.rows = [o.numpy() for o in s.out]
    return case, s


def run(state):
    case, s = state
    kind = case["kind"]
    if kind in ("fluid", "melt", "cg"):
        # a stretch of the run, then the state it reached
        s.run(case["steps"])
        s.read(s.rows)
        return {"pos": s.out[0], "vel": s.out[1], "force": s.out[2]}
    if kind == "replicas":
        call(s.lib, "espp_batch_run", s.b, case["steps"])
        for r, rows in zip(s.sys, s.rows):
            r.read(rows)
        return {"pos": s.out[0], "vel": s.out[1], "force": s.out[2]}
    if kind == "rdf":
        g = np.zeros(RDF_BINS)
        call(s.lib, "espp_rdf", s.h, RDF_BINS, dptr(g))
        return g
    if kind == "observables":
        e, w, k = ctypes.c_double(), np.zeros(6), np.zeros(6)
        call(s.lib, "espp_energy", s.h, _abi.IA_LJ, ctypes.byref(e))
        call(s.lib, "espp_virial_tensor", s.h, _abi.IA_LJ, dptr(w))
        call(s.lib, "espp_kinetic_tensor", s.h, dptr(k))
        return {"energy": e.value, "virial": w, "kinetic": k}
    # one frame of a training epoch: its forces against the target, the gradient, Adam
    loss = ctypes.c_double()
    call(s.lib, "espp_set_particles", s.h, s.n, i64ptr(s.ids), dptr(s.frame), None)
    call(s.lib, "espp_decompose", s.h)
    call(s.lib, "espp_mlp_fm_grad", s.h, s.n, i64ptr(s.ids), dptr(s.target), ctypes.byref(loss),
         dptr(s.grad))
    call(s.lib, "espp_mlp_adam_step", s.model, 1e-4, 0.9, 0.999, 1e-8, 1.0)
    call(s.lib, "espp_mlp_get_params", s.model, len(s.theta), dptr(s.theta))
    return {"loss": loss.value, "grad": s.grad.copy(), "theta": s.theta.copy()}


# ---- work and tolerance ------------------------------------------------------------------
def _neighbours(rho, rc):
    return 2.0 / 3.0 * math.pi * rc ** 3 * rho


def work(case):
    kind = case["kind"]
    if kind == "replicas":
        s = (case["smin"] + case["smax"]) / 2.0
        n, steps = case["count"] * s ** 3, case["steps"]
    else:
        n, steps = case["nx"] * case["ny"] * case["nz"], case.get("steps", 1)
    if kind in ("fluid", "replicas", "melt"):
        # a particle-step: state read and written (168 B, in reference arithmetic 192 B) and
        # 4 B for each pair within cutoff + skin; 24 operations a pair
        pairs = _neighbours(RHO_MELT, RC_WCA + SKIN) if kind == "melt" else _neighbours(RHO, RC + SKIN)
        base = 192.0 if case["precision"] == "fp64" else 168.0
        return {"bytes": steps * n * (base + 4.0 * pairs) + 72.0 * n, "flops": steps * n * 24.0 * pairs}
    if kind == "rdf":
        return {"bytes": 24.0 * n, "flops": 12.0 * n * (n - 1) / 2}
    if kind == "observables":
        p = _neighbours(RHO, RC + SKIN)
        return {"bytes": n * (24.0 * 2 + 4.0 * p), "flops": n * p * 40.0}
    p = 2 * _neighbours(RHO_CG, RC_CG)
    net = 2.0 * (MLP_K * MLP_H + MLP_H * MLP_H + MLP_H)
    if kind == "train":
        return {"bytes": n * (24.0 * 3 + 8.0 * p), "flops": n * (6 * net + p * MLP_K * 30.0)}
    return {"bytes": steps * n * (168.0 + 4.0 * p), "flops": steps * n * (2 * net + p * MLP_K * 20.0)}


def tolerance(case):
    """About four times what another order of the sums (other threads per particle) gives
    after two passes: a run is chaotic, so rounding grows along it.  The largest difference
    is a pair at the truncated cutoff that FP32 rounding puts on the other side."""
    kind = case["kind"]
    if kind == "rdf":
        return "exact"  # counts, each normalised by the same factor
    if kind == "observables":
        return {"rel": 1e-12}
    if kind == "train":
        return {"rel": 1e-2}  # BF16 products: 2.6e-3 from 64 bits
    if kind == "cg":
        return {"rel": 2e-4, "max": 2e-2}  # the forces of a BF16 network among others
    if case["precision"] == "fp64":
        return {"rel": 1e-11, "max": 1e-9}
    return {"rel": 4e-5, "max": 1e-2}


# ---- the same results in 64 bits -------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _min_image(d, box):
    return d - box * torch.round(d / box)


def _pair_list(x, box, rl):
    """Index pairs (i, j), each once, closer than rl under the minimum image."""
    dev, n = x.device, len(x)
    nc = [int(b / rl) for b in box.tolist()]
    if min(nc) < 3:
        out = []
        for a in range(0, n, 1024):
            d = _min_image(x[a:a + 1024, None] - x[None], box)
            i, j = torch.nonzero((d * d).sum(-1) < rl * rl, as_tuple=True)
            i = i + a
            out.append(torch.stack([i[i < j], j[i < j]]))
        return torch.cat(out, 1)
    q = x - box * torch.floor(x / box)
    c = [torch.clamp((q[:, k] / box[k] * nc[k]).long(), 0, nc[k] - 1) for k in range(3)]
    cell = c[0] + nc[0] * (c[1] + nc[1] * c[2])
    order = torch.argsort(cell)
    ncell = nc[0] * nc[1] * nc[2]
    count = torch.bincount(cell, minlength=ncell)
    start = torch.cumsum(count, 0) - count
    m = int(count.max())
    slot = torch.arange(n, device=dev) - start[cell[order]]
    table = torch.full((ncell, m), -1, dtype=torch.int64, device=dev)
    table[cell[order], slot] = order
    grid = torch.arange(ncell, device=dev)
    cx, cy, cz = grid % nc[0], (grid // nc[0]) % nc[1], grid // (nc[0] * nc[1])
    half = [(0, 0, 0)] + [(a, b, e) for e in (-1, 0, 1) for b in (-1, 0, 1) for a in (-1, 0, 1)
                          if (e, b, a) > (0, 0, 0)]
    out, chunk = [], max(1, 30_000_000 // (m * m))
    for ox, oy, oz in half:
        other = (cx + ox) % nc[0] + nc[0] * ((cy + oy) % nc[1] + nc[1] * ((cz + oz) % nc[2]))
        for a in range(0, ncell, chunk):
            ti, tj = table[a:a + chunk], table[other[a:a + chunk]]
            d = _min_image(x[ti][:, :, None] - x[tj][:, None], box)
            ok = ((d * d).sum(-1) < rl * rl) & (ti >= 0)[:, :, None] & (tj >= 0)[:, None]
            if (ox, oy, oz) == (0, 0, 0):
                ok &= ti[:, :, None] < tj[:, None]
            w, p, r = torch.nonzero(ok, as_tuple=True)
            out.append(torch.stack([ti[w, p], tj[w, r]]))
    return torch.cat(out, 1)


def _add_pairs(F, i, j, f):
    F.index_add_(0, i, f)
    F.index_add_(0, j, -f)


def _lj_forces(F, x, box, pairs, typ, terms):
    nt = max(k[1] for k in terms) + 1
    par = torch.zeros((nt, nt, 3), dtype=torch.float64, device=x.device)
    for (a, b), (eps, sig, rc) in terms.items():
        par[a, b] = par[b, a] = torch.tensor([48 * eps * sig ** 12, 24 * eps * sig ** 6, rc * rc],
                                             dtype=torch.float64)
    for a in range(0, pairs.shape[1], 40_000_000):
        i, j = pairs[0, a:a + 40_000_000], pairs[1, a:a + 40_000_000]
        d = _min_image(x[i] - x[j], box)
        r2 = (d * d).sum(-1)
        p = par[typ[i], typ[j]] if nt > 1 else par[0, 0].expand(len(i), 3)
        s = 1.0 / r2
        s6 = s * s * s
        ff = torch.where(r2 <= p[:, 2], s6 * (p[:, 0] * s6 - p[:, 1]) * s, 0.0)
        _add_pairs(F, i, j, d * ff[:, None])


def _tab(tab, x):
    """Linear interpolation of a table's force column."""
    r, _, f = (torch.as_tensor(a, device=x.device) for a in tab)
    k = torch.clamp(((x - r[0]) / (r[1] - r[0])).long(), 0, len(r) - 2)
    a = (f[k + 1] - f[k]) / (r[k + 1] - r[k])
    return a * (x - r[k]) + f[k]


def _mlp_energy(r_ij, i, j, n, theta, shift, scale):
    K, H = MLP_K, MLP_H
    w = (RC_CG - R0_CG) / (K - 1)
    mu = R0_CG + w * torch.arange(K, dtype=torch.float64, device=r_ij.device)
    fc = torch.where(r_ij < RC_CG, (torch.cos(math.pi * r_ij / RC_CG) + 1) / 2, 0.0)
    gk = torch.exp(-(r_ij[:, None] - mu) ** 2 / (2 * w * w)) * fc[:, None]
    G = torch.zeros((n, K), dtype=torch.float64, device=r_ij.device)
    G = G.index_add(0, i, gk).index_add(0, j, gk)
    W1, b1, W2, b2, w3, b3 = torch.split(theta, [H * K, H, H * H, H, H, 1])
    h = torch.nn.functional.silu((G - shift) * scale @ W1.view(H, K).T + b1)
    h = torch.nn.functional.silu(h @ W2.view(H, H).T + b2)
    return (h @ w3 + b3).sum()


def _mlp_forces(x, box, pairs, theta, shift, scale, create_graph=False):
    x = x.detach().requires_grad_(True)
    i, j = pairs
    r = torch.sqrt((_min_image(x[i] - x[j], box) ** 2).sum(-1))
    e = _mlp_energy(r, i, j, len(x), theta, shift, scale)
    return -torch.autograd.grad(e, x, create_graph=create_graph)[0]


def _uniforms(seed, ids, step, phase):
    """Philox4x32-10 keyed on the seed, counter (id, step, phase): three uniforms each."""
    m = 0xFFFFFFFF
    c = [ids & m, ids >> 32, torch.full_like(ids, step & m),
         torch.full_like(ids, ((step >> 32) & 0x7FFFFFFF) | (phase << 31))]
    k0, k1 = seed & m, (seed >> 32) & m

    def mul(a, b):  # 32 x 32 -> (high, low) without leaving 64 signed bits
        lo, hi = a * (b & 0xFFFF), a * (b >> 16)
        s = lo + ((hi & 0xFFFF) << 16)
        return ((hi >> 16) + (s >> 32)) & m, s & m

    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
        h0, l0 = mul(c[0], 0xD2511F53)
        h1, l1 = mul(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
    return torch.stack([(v.double() + 0.5) / 4294967296.0 for v in c[:3]], 1)


def _trajectory(case, seed):
    """Position, velocity and total force after the case's steps, in 64 bits."""
    dev = _dev()
    pos, vel, typ, box, g = _particles(case, seed)
    kind, n = case["kind"], len(pos)
    theta = torch.as_tensor(_mlp_params(g), device=dev) if kind == "cg" else None
    x, v, box = (torch.as_tensor(a, device=dev) for a in (pos, vel, box))
    typ = torch.as_tensor(typ, device=dev).long()
    x = x - torch.floor(x / box) * box
    rc = {"melt": RC_WCA, "cg": RC_CG}.get(kind, RC)
    m = 4.0 if kind == "cg" else 1.0
    ids = torch.arange(n, device=dev)
    lst = {"x": None}

    def forces():
        margin = 0.6
        if lst["x"] is None or float(_min_image(x - lst["x"], box).abs().max()) * math.sqrt(3) > margin / 2:
            lst["p"], lst["x"] = _pair_list(x, box, rc + margin), x.clone()
        F = torch.zeros_like(x)
        p = lst["p"]
        if kind != "cg":
            _lj_forces(F, x, box, p, typ, _lj_terms(case))
        if kind in ("melt", "cg"):
            b = torch.as_tensor(_bonds(n, case["beads"]), device=dev).T
            d = _min_image(x[b[0]] - x[b[1]], box)
            r2 = (d * d).sum(-1)
            r = torch.sqrt(r2)
            ff = -30.0 / (1.0 - r2 / 2.25) if kind == "melt" else _tab(_bond_table(), r) / r
            _add_pairs(F, b[0], b[1], d * ff[:, None])
        if kind == "cg":
            i, j = p
            d = _min_image(x[i] - x[j], box)
            r = torch.sqrt((d * d).sum(-1))
            ff = torch.where(r <= RC_CG, _tab(_pair_table(), r) / r, 0.0)
            _add_pairs(F, i, j, d * ff[:, None])
            t = torch.as_tensor(_triples(n, case["beads"]), device=dev).T
            d1, d3 = _min_image(x[t[0]] - x[t[1]], box), _min_image(x[t[2]] - x[t[1]], box)
            q1, q3 = (d1 * d1).sum(-1), (d3 * d3).sum(-1)
            c = (d1 * d3).sum(-1) / torch.sqrt(q1 * q3)
            a = (_tab(_angle_table(), torch.acos(c)) / torch.sqrt(1 - c * c))
            f1 = (a * c / q1)[:, None] * d1 - (a / torch.sqrt(q1 * q3))[:, None] * d3
            f3 = (a * c / q3)[:, None] * d3 - (a / torch.sqrt(q1 * q3))[:, None] * d1
            F.index_add_(0, t[0], f1).index_add_(0, t[2], f3).index_add_(0, t[1], -(f1 + f3))
            shift, scale = (torch.as_tensor(q, device=dev) for q in _mlp_norm())
            F += _mlp_forces(x, box, p, theta, shift, scale)
        return F

    dt, lang = _dynamics(case)

    def thermostat(F, step, phase):
        if not lang:
            return F
        amp = math.sqrt(24.0 * lang[1] * lang[0] / dt) * (math.sqrt(3.0) if phase else 1.0)
        return F - lang[0] * m * v + amp * (_uniforms(seed + 1, ids, step, phase) - 0.5) * math.sqrt(m)

    F = thermostat(forces(), 0, 1)
    v = v + 0.5 * dt / m * F
    moved = v * dt
    x = x + moved
    far = 0.0
    for step in range(case["steps"]):
        far += math.sqrt(float((moved * moved).sum(-1).max()))
        if far > SKIN / 2:  # the re-sort folds positions into the box
            x = x - torch.floor(x / box) * box
            far = 0.0
        F = thermostat(forces(), step, 0)
        v = v + 0.5 * dt / m * F
        if step + 1 < case["steps"]:
            v = v + 0.5 * dt / m * F
            moved = v * dt
            x = x + moved
    return x, v, F


def exact(case, seed):
    kind, dev = case["kind"], _dev()
    if kind in ("fluid", "melt", "cg"):
        x, v, F = _trajectory(case, seed)
        return {"pos": x, "vel": v, "force": F}
    if kind == "replicas":
        parts = [_trajectory(c, seed + 1000 * (k + 1))
                 for k, c in enumerate(_replica_cases(case))]
        return {name: torch.cat([p[q] for p in parts]) for q, name in enumerate(("pos", "vel", "force"))}
    pos, vel, typ, box, g = _particles(case, seed)
    x, box = torch.as_tensor(pos, device=dev), torch.as_tensor(box, device=dev)
    n = len(pos)
    x = x - torch.floor(x / box) * box
    if kind == "rdf":
        dr = float(box[1]) / 2 / RDF_BINS
        hist = torch.zeros(RDF_BINS, dtype=torch.int64, device=dev)
        for a in range(0, n, 1024):
            r = torch.sqrt((_min_image(x[a:a + 1024, None] - x[None], box) ** 2).sum(-1))
            k = torch.arange(n, device=dev)
            b = (r / dr).long()[k[a:a + 1024, None] < k[None]]
            hist += torch.bincount(b[b < RDF_BINS], minlength=RDF_BINS)
        rad = (np.arange(RDF_BINS) + 0.5) * dr
        rho = n / float(box.prod())
        return hist.cpu().numpy() / (2 * math.pi * dr * rho * n * (rad * rad + dr * dr / 12.0))
    if kind == "observables":
        i, j = _pair_list(x, box, RC)
        d = _min_image(x[i] - x[j], box)
        s6 = 1.0 / (d * d).sum(-1) ** 3
        q = RC ** -6.0
        e = (4.0 * (s6 * s6 - s6) - 4.0 * (q * q - q)).sum()
        f = d * (s6 * (48.0 * s6 - 24.0) / (d * d).sum(-1))[:, None]
        vel = torch.as_tensor(vel, device=dev)
        ax = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
        return {"energy": float(e), "virial": torch.stack([(d[:, a] * f[:, b]).sum() for a, b in ax]),
                "kinetic": torch.stack([(vel[:, a] * vel[:, b]).sum() for a, b in ax])}
    theta = torch.as_tensor(_mlp_params(g), device=dev).requires_grad_(True)
    target = torch.as_tensor(g.normal(0.0, 3.0, (n, 3)), device=dev)
    shift, scale = (torch.as_tensor(a, device=dev) for a in _mlp_norm())
    F = _mlp_forces(x, box, _pair_list(x, box, RC_CG), theta, shift, scale, create_graph=True)
    loss = ((F - target) ** 2).sum() / (3 * n)
    grad = torch.autograd.grad(loss, theta)[0]
    return {"loss": float(loss), "grad": grad.detach(), "theta": None}
