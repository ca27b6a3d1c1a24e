"""Performance cases: what a user's program has the framework do.

Two kinds of pass, both through the public model class:

* ``steps``  — one output interval of a simulation: the displacements,
  velocities and positions go in from pinned host buffers, a number of
  explicit time steps run on the device as replays of a step graph, and
  displacements, velocities, positions and force densities come back
  (``GpuDEMModel.step_host``).  Every pass holds whole contact-search
  intervals, so each pays for its list rebuilds.
* ``forces`` — one evaluation of the peridynamic forces on a given state
  (``GpuDEMModel.compute_pd_forces`` and the fields it writes), the call of a
  host that integrates by itself.

The mixed form evaluates bond forces in FP32, so its results are handed on as
FP32; the FP64 form's stay FP64.
"""
import functools
import math

import numpy as np
import torch

from peridem_b200 import scene as scn
from peridem_b200.model import PREC_FP64, PREC_MIXED, GpuDEMModel

LAWS = ("RNPBond", "PMBBond", "PDElasticBond", "PDState")
SEARCH_INTERVAL = 40  # steps between contact-list rebuilds of the named workloads
GRAPH_STEPS = 20      # steps per replayed graph


def _case(name, kind, shape, count, h_div, law, precision, scheme="central", steps=0, strain=2e-4, notch=False):
    c = dict(kind=kind, shape=shape, count=count, h_div=h_div, law=law, precision=precision, scheme=scheme,
             steps=steps, strain=strain, notch=notch)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest scene a user steps: two discs meeting (R / h = 10), the
        # drop-in FP64 form; every kernel is a few CTAs, launches count
        _case("pair_fp64", "steps", "pair", 2, 10, "RNPBond", "fp64", steps=200),
        # a two-disc impact study on a finer mesh with the prototype brittle
        # law and velocity Verlet, mixed form
        _case("pair_pmb_verlet_mixed", "steps", "pair", 2, 21, "PMBBond", "mixed", scheme="verlet", steps=200),
        # a small 2-D compression, as parameter studies run them by the hundred
        _case("pack43_mixed", "steps", "pack", 43, 13, "RNPBond", "mixed", steps=120),
        # the headline workload: 502 discs and hexagons at R / h = 15
        # compressed in a box, mixed form ...
        _case("pack502_mixed", "steps", "pack", 502, 15, "RNPBond", "mixed", steps=120),
        # ... and the same in the drop-in FP64 form
        _case("pack502_fp64", "steps", "pack", 502, 15, "RNPBond", "fp64", steps=40),
        # a large 2-D packing (the 2 000-particle workload's shapes and mesh)
        _case("pack2000_mixed", "steps", "pack", 2000, 15, "RNPBond", "mixed", steps=80),
        # a batched ensemble of compression scenes of uneven size
        _case("ensemble12_mixed", "steps", "ensemble", 12, 12, "RNPBond", "mixed", steps=80),
        # a 3-D column of spheres (R / h = 10) under a piston, state-based
        # law, mixed form (the 3-D workload's mesh, fewer spheres)
        _case("column48_state_mixed", "steps", "column", 48, 10, "PDState", "mixed", steps=40),
        # the same law and mesh in the drop-in FP64 form
        _case("column18_state_fp64", "steps", "column", 18, 10, "PDState", "fp64", steps=40),
        # one force evaluation of a cracked 2-D packing at a strain that
        # breaks bonds, mixed form
        _case("forces_pmb_notched_mixed", "forces", "pack", 330, 15, "PMBBond", "mixed", strain=3e-2, notch=True),
        # one force evaluation in 3-D, elastic bonds, FP64
        _case("forces_elastic3d_fp64", "forces", "column", 30, 8, "PDElasticBond", "fp64", strain=1e-3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    shape = rng.choice(["pair", "pack", "pack", "ensemble", "column"])
    kind = "steps" if shape == "ensemble" else rng.choice(["steps", "steps", "steps", "forces"])
    precision = rng.choice(["mixed", "fp64"])
    law = rng.choice(LAWS)
    if shape == "pair":
        count, h_div = 2, rng.randint(6, 24)
    elif shape == "pack":
        count, h_div = _log_int(rng, 12, 1200), rng.randint(8, 16)
    elif shape == "ensemble":
        count, h_div, law = rng.randint(2, 10), rng.randint(8, 12), "RNPBond"
    else:
        count, h_div = _log_int(rng, 4, 32), rng.randint(5, 10)
    steps = 0 if kind == "forces" else SEARCH_INTERVAL * (rng.randint(1, 5) if shape == "pair" else rng.randint(1, 2))
    scheme = rng.choice(["central", "central", "verlet"]) if kind == "steps" else "central"
    return _case("", kind, shape, count, h_div, law, precision, scheme, steps,
                 strain=rng.choice([1e-4, 2e-4, 1e-3]) if kind == "forces" else 2e-4,
                 notch=kind == "forces" and rng.random() < 0.5)


@functools.lru_cache(maxsize=4)
def _scene(shape, count, h_div, law, scheme):
    """The scene's geometry, materials and boundary conditions (made once; the
    seed makes the state)."""
    if shape == "pair":
        specs = [scn.two_particle(h_div=h_div, material=law, gap=0.02e-3 / h_div)]
    elif shape == "pack":
        # nearly equal bodies on a lattice just beyond the contact radius:
        # every neighbour is a contact candidate
        r = 1.25e-3
        per_row = max(3, int(round(math.sqrt(count / 2.0))))
        h = 0.96 * r / h_div
        specs = [scn.compressive_2d(count, r_range=(0.96 * r, r), h_div=h_div, material=law, gap=0.96 * h,
                                    width=(per_row + 0.6) * (2 * r + h), dt=5e-8)]
    elif shape == "ensemble":
        specs = scn.ensemble_specs(count, seed=1, h_div_range=(8, h_div), material=law)
    else:
        specs = [scn.column_3d(count, median_r=2e-3, sigma=0.1, h_div=h_div, material=law, wall_h=0.4e-3,
                               wall_layers=2.0, footprint=(3, 3) if count > 8 else (2, 2))]
    for s in specs:
        s.time_scheme = "velocity_verlet" if scheme == "verlet" else "central_difference"
    scenes = [scn.build_scene(s) for s in specs]
    return scenes[0] if len(scenes) == 1 else scn.merge_scenes(scenes)


def _of(case):
    return _scene(case["shape"], case["count"], case["h_div"], case["law"], case["scheme"])


def _motion(case, seed):
    """A state in mid-run: every body shifted by a few per cent of its mesh
    size (so that neighbours touch), strained as a whole, moving at about
    0.1 m/s and vibrating inside; walls at rest."""
    sc = _of(case)
    rng = np.random.default_rng(seed)
    dim, n = sc.dim, sc.n_particles
    moving = (sc.p_type == 0) & (sc.p_compute_force != 0)
    owner = sc.ptid.astype(np.int64)
    on = moving[owner][:, None]
    h = sc.p_h[owner][:, None]
    rel = sc.xref - sc.xref[sc.p_center][owner]
    e = rng.uniform(-1.0, 1.0, (n, 3, 3)) * case["strain"]
    e = 0.5 * (e + e.transpose(0, 2, 1))
    shift = rng.normal(0.0, 0.02, (n, 3))
    u = np.einsum("nab,nb->na", e[owner], rel) + h * (shift[owner] + 0.05 * case["strain"] * rng.normal(size=rel.shape))
    v = rng.normal(0.0, 0.1, (n, 3))[owner] + rng.normal(0.0, 0.05, rel.shape)
    u, v = np.where(on, u, 0.0), np.where(on, v, 0.0)
    u[:, dim:] = 0.0
    v[:, dim:] = 0.0
    return u, v


def _cut(sc):
    """Per node +1 or -1: the side of its body's notch it lies on (0 past the
    notch's tip); bonds that join the sides are broken before the call."""
    rel = sc.xref - sc.xref[sc.p_center][sc.ptid.astype(np.int64)]
    return np.where(rel[:, 0] < 0.0, np.where(rel[:, 1] > 0.1 * sc.p_h.min(), 1, -1), 0)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return t


def prepare(case, seed):
    sc = _of(case)
    u, v = _motion(case, seed)
    model = GpuDEMModel(sc, precision=PREC_MIXED if case["precision"] == "mixed" else PREC_FP64,
                        build_neighbors=True, compute_mx=True)
    state = {"case": case, "model": model}
    if case["kind"] == "forces":
        model.set_field("u", u)
        if case["notch"]:
            rp, col = model.pd_neighbors()
            side = _cut(sc)
            i = np.repeat(np.arange(sc.n_nodes), np.diff(rp.astype(np.int64)))
            model.set_field("bonds", (side[i] * side[col.astype(np.int64)] < 0).astype(np.uint8))
        return state
    model.integrate_begin()
    model.integrate_step(0, graph_steps=GRAPH_STEPS)  # captures the step graph, runs nothing
    state["host"] = {"u": _pinned(u), "v": _pinned(v), "x": _pinned(sc.xref + u), "f": _pinned(np.zeros_like(u))}
    state["views"] = {k: t.numpy() for k, t in state["host"].items()}
    return state


def run(state):
    case, model = state["case"], state["model"]
    mixed = case["precision"] == "mixed"
    if case["kind"] == "forces":
        model.compute_pd_forces()
        f = torch.from_numpy(model.field("f"))
        return {"f": f.float() if mixed else f, "Z": model.field("Z")}
    w = state["views"]
    model.step_host(w["u"], w["v"], w["x"], w["f"], case["steps"])
    return {k: t.float() if mixed else t for k, t in state["host"].items()}


def work(case):
    """Per step: each bond's neighbour index (4 B) and broken flag (1 bit) per
    end; per node its reference position, volume, displacement, velocity,
    position and force read, the last four written; once per pass the host
    buffers in and out.  A force evaluation: the bonds, reference position,
    displacement and volume read, force and damage written."""
    sc = _of(case)
    nodes = int(sum((sc.p_end - sc.p_start)[sc.p_compute_force != 0]))
    bonds = nodes * (22.4 if sc.dim == 2 else 87.0)
    vec = 8 * sc.dim
    flops = bonds * ({"RNPBond": 32, "PMBBond": 28, "PDElasticBond": 26, "PDState": 60}[case["law"]] + 8 * (sc.dim - 2))
    if case["kind"] == "forces":
        return {"bytes": bonds * 4.125 + nodes * (3 * vec + 12), "flops": flops}
    per_step = bonds * 4.125 + nodes * (9 * vec + 12)
    return {"bytes": case["steps"] * per_step + 7 * 24 * sc.n_nodes, "flops": case["steps"] * (flops + 30 * nodes)}


def _greater(a, b):
    """util::isGreater of the reference: a exceeds b beyond a relative 1e-5."""
    return (a - b) > 1e-5 * torch.maximum(a.abs(), b.abs())


def _body_forces(sc, p, law, x, u, vol, side):
    """Force density and damage of one body's nodes by the bond law, all pairs
    at once in FP64."""
    dim = sc.dim
    hor, h = float(sc.p_horizon[p]), float(sc.p_h[p])
    mat = [float(a) for a in sc.p_mat[p]]
    one = torch.ones((), dtype=torch.float64, device=x.device)
    dx = [x[None, :, a] - x[:, None, a] for a in range(dim)]
    r2 = sum(d * d for d in dx)
    bond = (r2 < hor * hor) & ~torch.eye(len(x), dtype=torch.bool, device=x.device)
    r = torch.where(bond, r2.sqrt(), one)
    du = [u[None, :, a] - u[:, None, a] for a in range(dim)]
    y = [a + b for a, b in zip(dx, du)]
    broken = bond & (side[None, :] * side[:, None] < 0)
    p0, p1 = (float(a) for a in sc.inf_params[:2])
    q = r / hor
    infl = p0 * torch.ones_like(q) if sc.inf_type == 0 else p0 + p1 * q if sc.inf_type == 1 else p0 * torch.exp(-q * q / p1)
    volj = vol[None, :].expand(len(x), -1)
    corr = torch.where(_greater(r, (hor - 0.5 * h) * one), volj * ((hor + 0.5 * h - r) / h), volj)
    if law == "RNPBond":
        ly = r
        s = sum(a * b for a, b in zip(dx, du)) / torch.where(bond, r2, one)
        sc_ = mat[2] / r.sqrt()
    else:
        ly = torch.where(bond, sum(a * a for a in y).sqrt(), one)
        s = (ly - r) / r
        sc_ = torch.full_like(r, {"PMBBond": mat[1], "PDState": mat[2]}.get(law, float(np.finfo(np.float64).max)))
    if law == "RNPBond" and mat[5] != 0.0:
        new = _greater(s.abs(), mat[4] * sc_)
    elif law in ("PMBBond", "PDState"):
        new = _greater(s.abs(), sc_ + 1e-10)
    else:
        new = torch.zeros_like(bond)
    gone = broken | new
    zero = torch.zeros_like(r)
    if law == "RNPBond":
        ef = infl * 4.0 * s * mat[0] * mat[1] * torch.exp(-mat[1] * r * s * s) / mat[3]
        axis = [a / r for a in dx]
    elif law == "PDState":
        K, G = mat[0], mat[1]
        m = torch.where(bond, r2 * infl * corr, zero).sum(1)
        th = 3.0 * torch.where(bond & ~gone, r * (ly - r) * infl * corr, zero).sum(1) / m
        a = 15.0 * G / m
        t = th * (3.0 * K / m - a / 3.0)
        ef = infl * (r * (t[:, None] + t[None, :]) + s * r * (a[:, None] + a[None, :]))
        axis = [b / ly for b in y]
    else:
        ef = infl * mat[0] * s
        axis = [b / ly for b in y]
    # a bond that breaks in this evaluation carries no force, except that the
    # state-based law breaks it in its pre-pass, ahead of the force loop
    hard = gone if law == "PDState" else broken
    live = torch.where(bond & ~gone, ef * corr, zero)
    ry = torch.where(bond, sum(a * a for a in y).sqrt(), one)
    push = torch.where(bond & hard, torch.clamp(float(sc.p_kn[p]) * volj * (ry - float(sc.p_rc[p])) / ry, max=0.0), zero)
    f = torch.zeros_like(x)
    for a in range(dim):
        f[:, a] = (live * axis[a] + push * y[a]).sum(1)
    return f, torch.where(bond, (s / sc_).abs(), zero).amax(1)


def exact(case, seed):
    """A force evaluation in FP64 from the definition of the laws; a pass of
    many steps has no such value."""
    if case["kind"] != "forces":
        return None
    sc = _of(case)
    u, _ = _motion(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    x, ud, vol = put(sc.xref), put(u), put(sc.vol)
    side = put(_cut(sc) if case["notch"] else np.zeros(sc.n_nodes, dtype=np.int64))
    f, z = torch.zeros_like(x), torch.zeros(sc.n_nodes, dtype=torch.float64, device=dev)
    for p in range(sc.n_particles):
        if not sc.p_compute_force[p]:
            continue
        k = slice(int(sc.p_start[p]), int(sc.p_end[p]))
        f[k], z[k] = _body_forces(sc, p, case["law"], x[k], ud[k], vol[k], side[k])
    return {"f": f.cpu(), "Z": z.cpu()}
