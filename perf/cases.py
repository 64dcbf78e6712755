"""Performance cases of the ring-polymer framework.

Every case is one call sequence of a user's program on the public API
(``DPM2D``, ``Batch``, ``diff``): upload a state, build the list, run, read the
result back.  The ranges are those of the repository's workloads
(``cudaring_b200/synth.py``, ``bench.py`` and the tests): 32 to 65,536
deformable rings of 16 to 45 vertices, rigid rings of 24 vertices, batches of
packings of 16 to 256 rings, FP64 and mixed precision, vertex-vertex and smooth
vertex-segment interactions, integration, minimisation and derivatives.

States are synthetic dense packings made on the host from the seed alone: ring
centres relaxed on a randomly occupied triangular lattice, every ring the
rounded power cell of its centre, sampled at equal arc length.  Facing rings
then sit at a chosen gap (in units of the sum of their vertex radii), as they
do in a compressed packing, and rest lengths, areas and angles are those of the
sampled shapes up to a small jitter, so that the shape terms start near rest.
The Hessian solves need a state that is stable, as a minimised packing is: equal
rings on the full lattice, the vertices of facing rings nested.

``exact`` restates the same physics in 64 bits with torch: the energy as a
plain function of the positions, forces and derivatives by autograd, the
integrators and FIRE as written in the reference.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cudaring_b200 import DPM2D, diff, synth
from cudaring_b200.batch import Batch
from cudaring_b200.dpm2d import simControl

WCA_CUT = 1.122462048
FIRE = [0.2, 0.5, 1.1, 0.99]  # a_start, f_dec, f_inc, f_a of the reference's drivers
FIRE_MIN_STEP = 20

# Constants of each kind of run: pair potential and interaction, shape
# constants (ea, el, eb), gap between facing rings in radius sums, jitter in
# rest lengths, time step, temperature, ring-size mix (nv small, nv large).
KINDS = {
    "force": dict(potential="harmonic", interaction="vertexVertex", ea=1.0, el=1.0, eb=0.01, gap=0.8, jitter=0.05,
                  dt=0.005, T=1e-3, nv=(16, 22)),
    "sample": dict(potential="harmonic", interaction="vertexVertex", ea=1.0, el=1.0, eb=0.01, gap=0.8, jitter=0.05,
                   dt=0.005, T=1e-3, nv=(16, 22)),
    "nve": dict(potential="lennardJones", interaction="vertexSmooth", ea=1e5, el=20.0, eb=10.0, gap=1.08,
                jitter=0.005, dt=0.002, T=0.01, nv=(32, 45)),
    "langevin": dict(potential="adhesive", interaction="vertexSmooth", ea=1e3, el=20.0, eb=1.0, gap=0.95, jitter=0.01,
                     dt=0.002, T=0.01, nv=(24, 33), l1=0.05, l2=0.2, gamma=1.0),
    "rigid": dict(potential="wca", interaction="vertexVertex", ea=0.0, el=0.0, eb=0.0, gap=1.0, jitter=0.0, dt=0.001,
                  T=0.1, nv=(24, 24), gamma=1.0, driving=0.1, taup=100.0),
    "fire": dict(potential="harmonic", interaction="vertexVertex", ea=1.0, el=1.0, eb=0.01, gap=0.8, jitter=0.05,
                 dt=1e-2, T=0.0, nv=(16, 22)),
    "batch_fire": dict(potential="harmonic", interaction="vertexVertex", ea=1.0, el=1.0, eb=0.01, gap=0.8, jitter=0.05,
                       dt=1e-2, T=0.0, nv=(16, 22)),
    "solve": dict(potential="harmonic", interaction="vertexVertex", ea=1.0, el=1.0, eb=0.5, gap=0.77, jitter=0.01,
                  dt=0.002, T=0.0, nv=(33, 33), crystal=True),
    "adjoint": dict(potential="harmonic", interaction="vertexVertex", ea=1.0, el=1.0, eb=0.01, gap=0.8, jitter=0.01,
                    dt=0.002, T=1e-4, nv=(32, 32)),
}


def listed():
    return [
        # one force evaluation of a small packing with new positions (what a
        # host-side minimiser or a test does per evaluation): call latency
        {"name": "force_32", "kind": "force", "rings": 32},
        # the small NVE run of 32 rings (608 vertices), energies sampled every
        # 50 steps as the reference's drivers do
        {"name": "sample_nve_32", "kind": "sample", "rings": 32, "steps": 500, "every": 50},
        # the 39,424-vertex Lennard-Jones run (1024 rings, nv 32/45) in FP64
        {"name": "nve_lj_1024", "kind": "nve", "rings": 1024, "steps": 200, "tile": 1, "precision": "fp64"},
        # the same in mixed precision
        {"name": "nve_lj_1024_mixed", "kind": "nve", "rings": 1024, "steps": 200, "tile": 1, "precision": "mixed"},
        # the scale-up: 8 x 8 periodic copies, 65,536 rings, 2.5M vertices
        {"name": "nve_lj_65536", "kind": "nve", "rings": 1024, "steps": 20, "tile": 8, "precision": "fp64"},
        # a thermostatted run of cohesive cells, ragged sizes
        {"name": "langevin_adhesive_333", "kind": "langevin", "rings": 333, "steps": 200},
        # rigid bumpy rings, 4096 x 24 vertices, Langevin in FP64
        {"name": "rigid_4096", "kind": "rigid", "rings": 4096, "steps": 100, "precision": "fp64", "active": False},
        # active rigid rings in mixed precision, fewer and ragged
        {"name": "rigid_active_1501_mixed", "kind": "rigid", "rings": 1501, "steps": 100, "precision": "mixed",
         "active": True},
        # FIRE after a compression step of one packing
        {"name": "fire_513", "kind": "fire", "rings": 513, "steps": 200},
        # FIRE of many packings of uneven size at once (compression to jamming)
        {"name": "batch_fire_96", "kind": "batch_fire", "systems": 96, "rings_min": 16, "rings_max": 256, "steps": 100},
        # linear response at a packing: a Hessian product and a budgeted
        # conjugate-gradient solve, 256 rings of 32
        {"name": "hessian_solve_256", "kind": "solve", "rings": 256, "steps": 64},
        # backward pass: gradients of an NVE trajectory by the adjoint
        {"name": "nve_adjoint_256", "kind": "adjoint", "rings": 256, "steps": 20, "every": 10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["force", "sample", "nve", "nve", "langevin", "rigid", "fire", "batch_fire", "solve", "adjoint"])
    if kind == "force":
        return {"kind": kind, "rings": _log_int(rng, 20, 4000)}
    if kind == "sample":
        return {"kind": kind, "rings": _log_int(rng, 16, 1500), "steps": rng.randrange(100, 300),
                "every": rng.choice([1, 10, 50, 77])}
    if kind == "nve":
        return {"kind": kind, "rings": _log_int(rng, 24, 2500), "steps": rng.randrange(20, 100),
                "tile": rng.choice([1, 1, 1, 2, 3]), "precision": rng.choice(["fp64", "fp64", "mixed"])}
    if kind == "langevin":
        return {"kind": kind, "rings": _log_int(rng, 30, 3000), "steps": rng.randrange(30, 100)}
    if kind == "rigid":
        return {"kind": kind, "rings": _log_int(rng, 60, 4096), "steps": rng.randrange(30, 100),
                "precision": rng.choice(["fp64", "mixed"]), "active": rng.random() < 0.5}
    if kind == "fire":
        return {"kind": kind, "rings": _log_int(rng, 20, 3000), "steps": rng.randrange(60, 200)}
    if kind == "batch_fire":
        return {"kind": kind, "systems": _log_int(rng, 3, 96), "rings_min": 16, "rings_max": rng.randrange(20, 256),
                "steps": rng.randrange(50, 110)}
    if kind == "solve":
        return {"kind": kind, "rings": _log_int(rng, 20, 700), "steps": rng.randrange(16, 64)}
    return {"kind": "adjoint", "rings": _log_int(rng, 20, 500), "steps": rng.randrange(8, 24), "every": rng.randrange(4, 12)}


# ------------------------------------------------------------------- packings
def _pairs(x, box, r):
    """Ordered pairs (i, j), i != j, of points closer than r in a periodic box."""
    n = len(x)
    nc = np.maximum(1, np.floor(box / r).astype(int))
    if nc.min() < 3:
        nc[:] = 1
    w = x - box * np.floor(x / box)
    c = np.minimum((w / box * nc).astype(int), nc - 1)
    cell = c[:, 1] * nc[0] + c[:, 0]
    order = np.argsort(cell, kind="stable")
    cnt = np.bincount(cell, minlength=nc[0] * nc[1])
    start = np.concatenate([[0], np.cumsum(cnt)])
    table = np.full((len(cnt), cnt.max()), -1)
    table[cell[order], np.arange(n) - start[cell[order]]] = order
    out_i, out_j = [], []
    span = (0,) if nc[0] == 1 else (-1, 0, 1)
    for dy in span:
        for dx in span:
            near = ((c[:, 1] + dy) % nc[1]) * nc[0] + (c[:, 0] + dx) % nc[0]
            cand = table[near]
            i, k = np.nonzero((cand >= 0) & (cand != np.arange(n)[:, None]))
            j = cand[i, k]
            d = w[i] - w[j]
            d -= box * np.round(d / box)
            ok = (d * d).sum(1) < r * r
            out_i.append(i[ok])
            out_j.append(j[ok])
    i, j = np.concatenate(out_i), np.concatenate(out_j)
    order = np.lexsort((j, i))
    return i[order], j[order]


def _lattice(n):
    """Columns and (even) rows of a triangular lattice with at least n sites, few vacant."""
    best = None
    for nx in range(2, 4 * int(math.sqrt(n)) + 4):
        ny = 2 * max(1, math.ceil(n / nx / 2))
        cost = (nx * ny - n) / n + 0.3 * abs(math.log(nx / (ny * math.sqrt(0.75))))
        if best is None or cost < best[0]:
            best = (cost, nx, ny)
    return best[1], best[2]


def _packing(n, k, seed):
    """A dense packing of n rings, half of each size (see the module's text)."""
    rng = np.random.default_rng(seed)
    crystal = k.get("crystal", False)
    nx, ny = _lattice(n)
    if crystal:
        n = nx * ny
    nv = np.array([k["nv"][0]] * (n // 2) + [k["nv"][1]] * (n - n // 2), dtype=np.int64)
    R = np.where(nv == k["nv"][0], 1.0, 1.4 if k["nv"][0] != k["nv"][1] else 1.0) / math.sqrt(math.pi)
    a = math.sqrt(np.mean(math.pi * R * R) / 0.93 * n / (nx * ny) / math.sqrt(0.75))
    box = np.array([nx * a, ny * a * math.sqrt(0.75)])
    site = rng.permutation(nx * ny)[:n]
    iy, ix = site // nx, site % nx
    x = np.stack([(ix + 0.5 * (iy % 2)) * a, iy * a * math.sqrt(0.75)], axis=1)
    if not crystal:
        x = x + rng.normal(0.0, 0.08 * a, (n, 2))
    for sweep in range(0 if crystal else 60):  # soft repulsion of the discs
        if sweep % 20 == 0:
            i, j = _pairs(x, box, 2.6 * R.max())
        d = x[i] - x[j]
        d -= box * np.round(d / box)
        r = np.sqrt((d * d).sum(1))
        f = (0.25 * np.maximum(0.0, 1.02 * (R[i] + R[j]) - r) / r)[:, None] * d
        x = x + np.stack([np.bincount(i, f[:, 0], n), np.bincount(i, f[:, 1], n)], axis=1)
    # rounded power cell of every ring: a soft minimum over its neighbours' faces
    i, j = _pairs(x, box, 3.6 * R.max())
    rad = math.pi * R / nv  # half the spacing of the vertices, nearly
    d = x[j] - x[i]
    d -= box * np.round(d / box)
    r = np.sqrt((d * d).sum(1))
    face = 0.5 * r + (R[i] ** 2 - R[j] ** 2) / (2.0 * r) - 0.5 * k["gap"] * (rad[i] + rad[j])
    slot = np.arange(len(i)) - np.searchsorted(i, i)
    most = int(slot.max()) + 1
    px, py = np.zeros((n, most)), np.zeros((n, most))
    px[i, slot] = d[:, 0] / (r * np.maximum(face, 0.2 * R[i]))
    py[i, slot] = d[:, 1] / (r * np.maximum(face, 0.2 * R[i]))
    m = 96
    th = 2.0 * math.pi * np.arange(m) / m
    inv = np.repeat((1.0 / (1.12 * R) ** 16)[:, None], m, axis=1)
    for s in range(most):
        c = np.maximum(0.0, px[:, s, None] * np.cos(th) + py[:, s, None] * np.sin(th))
        inv += (((c * c) ** 2) ** 2) ** 2
    rho = inv ** (-1.0 / 16.0)
    outline = np.stack([rho * np.cos(th), rho * np.sin(th)], axis=2)
    outline = np.concatenate([outline, outline[:, :1]], axis=1)
    arc = np.concatenate([np.zeros((n, 1)), np.cumsum(np.linalg.norm(np.diff(outline, axis=1), axis=2), axis=1)], axis=1)
    first = np.concatenate([[0], np.cumsum(nv)[:-1]])
    ring = np.repeat(np.arange(n), nv)
    frac = (np.arange(len(ring)) - first[ring] + (0.0 if crystal else rng.random(n)[ring])) / nv[ring]
    flat = (arc / arc[:, -1:]) * 0.5 + np.arange(n)[:, None]  # rows one after another, increasing
    at = np.searchsorted(flat.reshape(-1), frac * 0.5 + ring, side="right") - 1 - ring * (m + 1)
    at = np.clip(at, 0, m - 1)
    u = (frac * 0.5 + ring - flat[ring, at]) / (flat[ring, at + 1] - flat[ring, at])
    pos = x[ring] + outline[ring, at] * (1 - u)[:, None] + outline[ring, at + 1] * u[:, None]
    prev, nxt = _neighbours_in_ring(nv)
    seg = pos[nxt] - pos
    length = np.linalg.norm(seg, axis=1)
    l0 = (np.bincount(ring, length) / nv)[ring]
    rel = pos - pos[first[ring]]
    reln = pos[nxt] - pos[first[ring]]
    a0 = 0.5 * np.bincount(ring, rel[:, 0] * reln[:, 1] - rel[:, 1] * reln[:, 0])
    ps = seg[prev]
    theta0 = np.arctan2(seg[:, 0] * ps[:, 1] - seg[:, 1] * ps[:, 0], (seg * ps).sum(1))
    pos = pos + k["jitter"] * l0[:, None] * rng.uniform(-1.0, 1.0, pos.shape)
    vel = rng.normal(0.0, math.sqrt(k["T"]), (n, 2))[ring] if k["T"] > 0 else np.zeros_like(pos)
    return synth.Packing(nv_list=nv, pos=pos.reshape(-1).copy(), vel=vel.reshape(-1).copy(), rad=0.5 * l0, l0=l0,
                         theta0=theta0, a0=a0, box=box, centres=x)


def _neighbours_in_ring(nv):
    first = np.concatenate([[0], np.cumsum(nv)[:-1]])
    ring = np.repeat(np.arange(len(nv)), nv)
    at = np.arange(len(ring)) - first[ring]
    return first[ring] + (at - 1) % nv[ring], first[ring] + (at + 1) % nv[ring]


def _tiled(pk, t, seed, T):
    """t x t periodic copies of a packing, each ring with its own velocity."""
    if t == 1:
        return pk
    shift = [np.array([ix * pk.box[0], iy * pk.box[1]]) for iy in range(t) for ix in range(t)]
    pos = np.concatenate([(pk.pos.reshape(-1, 2) + s).reshape(-1) for s in shift])
    nv = np.tile(pk.nv_list, t * t)
    vel = np.random.default_rng(seed + 77).normal(0.0, math.sqrt(T), (len(nv), 2))
    rep = {f: np.tile(getattr(pk, f), t * t) for f in ("rad", "l0", "theta0", "a0")}
    return synth.Packing(nv_list=nv, pos=pos, vel=np.repeat(vel, nv, axis=0).reshape(-1), box=pk.box * t,
                         centres=np.zeros((len(nv), 2)), **rep)


def _inputs(case, seed):
    """The case's packings (a batch has several) and constants."""
    k = KINDS[case["kind"]]
    if case["kind"] == "batch_fire":
        # uneven ring counts, the same for every seed
        sizes = np.random.default_rng(case["systems"]).integers(case["rings_min"], case["rings_max"] + 1, case["systems"])
        return [_packing(int(n), k, seed + 1000 * s) for s, n in enumerate(sizes)], k
    pk = _packing(case["rings"], k, seed)
    return [_tiled(pk, case.get("tile", 1), seed, k["T"])], k


def _right_hand_side(case, seed, n):
    return np.random.default_rng(seed + 9).normal(0.0, 1.0, n)


# ----------------------------------------------------------------- the calls
def prepare(case, seed):
    packings, k = _inputs(case, seed)
    pair = {f: k[f] for f in ("potential", "interaction", "ea", "el", "eb", "l1", "l2") if f in k}
    s = {"case": case, "k": k}
    if case["kind"] == "batch_fire":
        b = Batch.from_packings(packings, **pair)
        b.setDisplacementCutoff(0.5)
        s.update(d=b, pos=b.getVertexPositions(), vel=np.zeros(2 * b.nv), sigma=b.getMeanParticleSizes())
        return s
    pk = packings[0]
    d = DPM2D.from_packing(pk, dt=k["dt"], **pair)
    cut = d.setDisplacementCutoff(0.5, 2.0 * float(pk.rad.mean()))
    s.update(d=d, pos=pk.pos, vel=pk.vel, cut=cut)
    if "precision" in case:
        d.setPrecision(case["precision"])
    if case["kind"] == "rigid":
        d.setShapeType(simControl.shapeEnum.rigid)
        if case["active"]:
            d.setParticleType(simControl.particleEnum.active)
            d.setSelfPropulsionParams(k["driving"], k["taup"])
        first = np.concatenate([[0], np.cumsum(pk.nv_list)[:-1]])
        s["vel"] = pk.vel.reshape(-1, 2)[first].reshape(-1).copy()
    if case["kind"] in ("langevin", "rigid"):
        s["seed"] = 1234 + seed % 1000
    if case["kind"] == "sample":
        d.calcNeighborList(cut)
        d.calcForceEnergy()
        d.initNVE(k["T"], readState=True)
    if case["kind"] == "solve":
        s["b"] = _right_hand_side(case, seed, 2 * d.numVertices)
    return s


def run(s):
    return globals()["_run_" + s["case"]["kind"]](s["d"], s, s["case"], s["k"])


def _upload(d, s):
    d.setVertexPositions(s["pos"])
    if s["case"]["kind"] == "rigid":
        d.setParticleVelocities(s["vel"])
    else:
        d.setVertexVelocities(s["vel"])
    d.calcNeighborList(s["cut"])


def _result(d):
    return {"pos": d.getVertexPositions(), "vel": d.getVertexVelocities(), "energy": d.getEnergy()}


def _run_force(d, s, case, k):
    d.setVertexPositions(s["pos"])
    d.calcNeighborList(s["cut"])
    d.calcForceEnergy()
    return {"force": d.getVertexForces(), "energy": d.getPotentialEnergy()}


def _run_sample(d, s, case, k):
    _upload(d, s)
    d.resetLastPositions()
    d.calcForceEnergy()
    energies = []
    for done in range(0, case["steps"], case["every"]):
        d.NVELoop(min(case["every"], case["steps"] - done))
        energies.append(d.getEnergy())
    return {"pos": d.getVertexPositions(), "vel": d.getVertexVelocities(), "energies": np.array(energies)}


def _run_nve(d, s, case, k):
    _upload(d, s)
    d.calcForceEnergy()
    d.initNVE(k["T"], readState=True)
    d.NVELoop(case["steps"])
    return _result(d)


def _run_langevin(d, s, case, k):
    _upload(d, s)
    d.calcForceEnergy()
    d.setSeed(s["seed"])
    d.initLangevin(k["T"], k["gamma"], readState=True)
    d.langevinLoop(case["steps"])
    return _result(d)


def _run_rigid(d, s, case, k):
    _upload(d, s)
    d.setSeed(s["seed"])
    d.initRigidLangevin(k["T"], k["gamma"], readState=True)
    d.rigidLangevinLoop(case["steps"])
    return {"pos": d.getVertexPositions(), "vel": d.getParticleVelocities(), "spin": d.getParticleAngularVelocities()}


def _run_fire(d, s, case, k):
    _upload(d, s)
    d.calcForceEnergy()
    d.initFIRE(FIRE + [k["dt"], 10 * k["dt"], 0.2], FIRE_MIN_STEP, 0, d.numVertices)
    iterations, _ = d.minimizeFIRE(1e-14, case["steps"])
    return dict(_result(d), iterations=iterations)


def _run_batch_fire(b, s, case, k):
    b.setVertexPositions(s["pos"])
    b.setVertexVelocities(s["vel"])
    b.calcNeighborLists()
    b.initFIRE(FIRE + [k["dt"], 10 * k["dt"], 0.2], FIRE_MIN_STEP, dt=k["dt"] * s["sigma"])
    iterations, _ = b.fireMinimize(1e-14, case["steps"])
    return {"pos": b.getVertexPositions(), "vel": b.getVertexVelocities(), "energies": b.getPotentialEnergies(),
            "iterations": iterations}


def _run_solve(d, s, case, k):
    d.setVertexPositions(s["pos"])
    d.calcNeighborList(s["cut"])
    x, iterations, _ = d.hessianSolve(s["b"], tol=1e-10, maxIter=case["steps"])
    return {"product": d.hvp(s["b"]), "solution": x, "iterations": iterations}


def _run_adjoint(d, s, case, k):
    value, gx, gv = diff.nve_gradient(d, s["pos"], s["vel"], case["steps"], k["dt"], checkpoint=case["every"])
    return {"value": value, "dx": gx, "dv": gv}


def work(case):
    """Inputs read once and outputs written once; operations of the physics:
    about 120 per vertex and step for the shape terms and the update, 35 for
    each of the few pair terms that act on it."""
    k = KINDS[case["kind"]]
    rings = case.get("rings", 0) * case.get("tile", 1) ** 2
    if case["kind"] == "batch_fire":
        rings = case["systems"] * (case["rings_min"] + case["rings_max"]) // 2
    nv = rings * sum(k["nv"]) // 2
    per_step = 120 + 35 * (4 if k["interaction"] == "vertexSmooth" else 2)
    steps = case.get("steps", 1)
    if case["kind"] in ("solve", "adjoint"):
        per_step *= 3  # the product of the Hessian with a vector
    # read: positions, velocities, radii, rest lengths and angles, areas; written: positions (or forces), velocities
    return {"bytes": 56 * nv + 8 * rings + 32 * nv, "flops": nv * per_step * steps}


# ------------------------------------------------------------ the same in 64 bits
class _Exact:
    """Energy, forces and sums of the given packings in float64 with torch."""

    def __init__(self, packings, k, skin):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda v, ty=torch.float64: torch.as_tensor(np.concatenate(v), dtype=ty, device=dev)  # noqa: E731
        self.k, self.dev = k, dev
        nvs = [p.nv_list for p in packings]
        off = np.concatenate([[0], np.cumsum([int(v.sum()) for v in nvs])])
        roff = np.concatenate([[0], np.cumsum([len(v) for v in nvs])])
        ring = [np.repeat(np.arange(len(v)), v) for v in nvs]
        nb = [_neighbours_in_ring(v) for v in nvs]
        firsts = [np.concatenate([[0], np.cumsum(v)[:-1]]) for v in nvs]
        self.ring = t([r + roff[s] for s, r in enumerate(ring)], torch.long)
        self.prev = t([b[0] + off[s] for s, b in enumerate(nb)], torch.long)
        self.next = t([b[1] + off[s] for s, b in enumerate(nb)], torch.long)
        self.first = t([firsts[s][ring[s]] + off[s] for s in range(len(nvs))], torch.long)
        self.system = t([np.full(off[s + 1] - off[s], s) for s in range(len(nvs))], torch.long)
        self.nvr, self.np, self.nv, self.S = t(nvs), int(roff[-1]), int(off[-1]), len(nvs)
        self.box = t([np.tile(p.box, (p.num_vertices, 1)) for p in packings])
        self.rad, self.l0 = t([p.rad for p in packings]), t([p.l0 for p in packings])
        self.theta0, self.a0 = t([p.theta0 for p in packings]), t([p.a0 for p in packings])
        self.x, self.v = (t([getattr(p, f).reshape(-1, 2) for p in packings]) for f in ("pos", "vel"))
        self.range = {"harmonic": 1.0, "lennardJones": 2.5, "wca": WCA_CUT, "adhesive": 1.0 + k.get("l2", 0.0)}[k["potential"]]
        smooth = 1.0 if k["interaction"] == "vertexSmooth" else 0.0
        i, j = [], []
        for s, p in enumerate(packings):
            a, b = _pairs(p.pos.reshape(-1, 2), p.box, 2.0 * p.rad.max() * (self.range + smooth) + skin)
            ok = ring[s][a] != ring[s][b]
            i.append(a[ok] + off[s])
            j.append(b[ok] + off[s])
        self.i, self.j = t(i, torch.long), t(j, torch.long)

    def wrap(self, d, at):
        L = self.box[at]
        return d - L * torch.round(d / L).detach()

    def pair(self, d, rsum):
        """Full pair energy at distance d within the range."""
        k = self.k
        if k["potential"] == "harmonic":
            return 0.5 * (1.0 - d / rsum) ** 2
        if k["potential"] == "adhesive":
            ov, l1, l2 = 1.0 - d / rsum, k["l1"], k["l2"]
            return torch.where(d < (1.0 + l1) * rsum, 0.5 * (ov * ov - l1 * l2), -0.5 * l1 / (l2 - l1) * (ov + l2) ** 2)
        r6 = (rsum / d) ** 6
        if k["potential"] == "wca":
            return 4.0 * (r6 * r6 - r6) + 1.0
        c6 = 2.5 ** -6
        shift = abs(24.0 * (2.0 * c6 - 1.0) * c6 / 2.5) / rsum
        return 4.0 * (r6 * r6 - r6) - 4.0 * (c6 * c6 - c6) - shift * (d - 2.5 * rsum)

    def inside(self, d, rsum):
        return d < rsum * self.range if self.k["potential"] in ("harmonic", "adhesive") else d <= rsum * self.range

    def add(self, out, where, values):
        return out.index_add(0, where, values)

    def energies(self, x):
        """Potential energy per system."""
        k, zero = self.k, torch.zeros(self.S, dtype=torch.float64, device=self.dev)
        ns = self.wrap(x[self.next] - x, slice(None))
        ps = ns[self.prev]
        u, un = self.wrap(x - x[self.first], slice(None)), self.wrap(x[self.next] - x[self.first], slice(None))
        sh = u[:, 0] * un[:, 1] - un[:, 0] * u[:, 1]
        area = 0.5 * self.add(torch.zeros(self.np, dtype=torch.float64, device=self.dev), self.ring, sh).abs()
        of_ring = 0.5 * k["ea"] * (area / self.a0 - 1.0) ** 2
        theta = torch.atan2(ns[:, 0] * ps[:, 1] - ns[:, 1] * ps[:, 0], (ns * ps).sum(1))
        e = (of_ring / self.nvr)[self.ring] + 0.5 * k["el"] * (ns.norm(dim=1) / self.l0 - 1.0) ** 2
        e = e + 0.5 * k["eb"] * (theta - self.theta0) ** 2
        out = self.add(zero, self.system, e)
        if k["interaction"] == "vertexVertex":
            return self.pairs_energy(x, out)
        return self.units_energy(x, ns, ps, out)

    def pairs_energy(self, x, out):
        with torch.no_grad():
            d = self.wrap(x[self.i] - x[self.j], self.i).norm(dim=1)
            on = (self.inside(d, self.rad[self.i] + self.rad[self.j]) & (self.i < self.j)).nonzero()[:, 0]
        i, j = self.i[on], self.j[on]
        d = self.wrap(x[i] - x[j], i).norm(dim=1)
        return self.add(out, self.system[i], self.pair(d, self.rad[i] + self.rad[j]))

    def units_energy(self, x, ns, ps, out):
        """Vertex i against the segment prev(j) -> j, with the corner terms."""
        with torch.no_grad():
            q = self.prev[self.j]
            tq, seg, pseg = self.wrap(x[self.i] - x[q], self.i), ns[q], ps[q]
            proj, pc = (tq * seg).sum(1) / (seg * seg).sum(1), (tq * pseg).sum(1)
            cross = (seg[:, 0] * tq[:, 1] - seg[:, 1] * tq[:, 0]).abs() / seg.norm(dim=1)
            rsum = self.rad[self.i] + self.rad[self.j]
            span = (proj >= 0) & (proj < 1)
            near = self.inside(tq.norm(dim=1), rsum)
            on = (span & self.inside(cross, rsum)).nonzero()[:, 0]
            convex = ~span & (proj < 0) & (pc >= 0) & near
            concave = span & (pc >= -(pseg * pseg).sum(1)) & (pc < 0) & near
            corner = (convex | concave).nonzero()[:, 0]
            sign = torch.where(convex[corner], 1.0, -1.0).to(torch.float64)
        i, q, seg = self.i[on], self.prev[self.j[on]], ns[self.prev[self.j[on]]]
        tq = self.wrap(x[i] - x[q], i)
        d = (seg[:, 0] * tq[:, 1] - seg[:, 1] * tq[:, 0]).abs() / seg.norm(dim=1)
        out = self.add(out, self.system[i], self.pair(d, rsum[on]))
        i, q = self.i[corner], self.prev[self.j[corner]]
        d = self.wrap(x[i] - x[q], i).norm(dim=1)
        return self.add(out, self.system[i], sign * self.pair(d, rsum[corner]))

    def force(self, x, energy=False):
        y = x.detach().requires_grad_(True)
        e = self.energies(y)
        f = -torch.autograd.grad(e.sum(), y)[0]
        return (f, e.detach()) if energy else f

    def per_system(self, values):
        return self.add(torch.zeros(self.S, dtype=torch.float64, device=self.dev), self.system, values)


def _host(t):
    return t.detach().cpu().numpy().reshape(-1)


def _normals(seed, stream, n):
    """Two normals per index from Philox4x32-10 (Salmon et al., SC'11) by Box-Muller, as the framework documents its streams."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [np.arange(n, dtype=np.uint64), np.zeros(n, np.uint64), np.full(n, stream & 0xFFFFFFFF, np.uint64),
         np.full(n, stream >> 32, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    a, b = (c[0] | (c[1] << np.uint64(32))) >> np.uint64(11), (c[2] | (c[3] << np.uint64(32))) >> np.uint64(11)
    r = np.sqrt(-2.0 * np.log((a.astype(float) + 0.5) / 2.0 ** 53))
    u = 2.0 * math.pi * b.astype(float) / 2.0 ** 53
    return np.stack([r * np.cos(u), r * np.sin(u)], axis=1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "nve" and case.get("tile", 1) > 3:
        return None  # 2.5 million vertices: over the time for this
    if kind == "rigid" and case["active"]:
        return None  # the propulsion angles start from the framework's own draw
    packings, k = _inputs(case, seed)
    skin = {"force": 0.0, "solve": 0.0, "adjoint": 0.02, "rigid": 0.3}.get(kind, 0.25)
    w = _Exact(packings, k, skin)
    x, v, dt = w.x, w.v, k["dt"]
    if kind == "force":
        f, e = w.force(x, energy=True)
        return {"force": _host(f), "energy": float(e.sum())}
    if kind == "solve":
        return _exact_solve(w, case, seed)
    if kind == "adjoint":
        return _exact_adjoint(w, case)
    if kind in ("fire", "batch_fire"):
        return _exact_fire(w, case, k)
    if kind == "rigid":
        return _exact_rigid(w, case, seed)
    f, energies = w.force(x), []
    every = case.get("every", case["steps"])
    noise = math.sqrt(2.0 * k["T"] * k["gamma"] / dt) if kind == "langevin" else 0.0
    kick = f  # the force of the half kick that opens a step
    for n in range(case["steps"]):
        v = v + 0.5 * dt * kick
        x = x + dt * v
        f, e = w.force(x, energy=True)
        kick = f
        if kind == "langevin":
            z = torch.as_tensor(_normals(1234 + seed % 1000, 2 * n, w.np), device=w.dev)[w.ring]
            kick = f + noise * z - k["gamma"] * v
        v = v + 0.5 * dt * kick
        if (n + 1) % every == 0 or n + 1 == case["steps"]:
            energies.append(float(e.sum() + 0.5 * (v * v).sum()))
    if kind == "sample":
        return {"pos": _host(x), "vel": _host(v), "energies": np.array(energies)}
    return {"pos": _host(x), "vel": _host(v), "energy": energies[-1]}


def _exact_solve(w, case, seed):
    b = torch.as_tensor(_right_hand_side(case, seed, 2 * w.nv).reshape(-1, 2), device=w.dev)
    x = w.x.detach().requires_grad_(True)
    f = torch.autograd.grad(w.energies(x).sum(), x, create_graph=True)[0]
    hb = torch.autograd.grad((f * b).sum(), x)[0]
    return {"product": _host(hb), "solution": None, "iterations": None}


def _exact_adjoint(w, case):
    dt = w.k["dt"]
    x0, v0 = w.x.clone().requires_grad_(True), w.v.clone().requires_grad_(True)
    grad = lambda y: -torch.autograd.grad(w.energies(y).sum(), y, create_graph=True)[0]  # noqa: E731
    x, v = x0, v0
    f = grad(x)
    for _ in range(case["steps"]):
        h = v + 0.5 * dt * f
        x = x + dt * h
        f = grad(x)
        v = h + 0.5 * dt * f
    value = w.energies(x).sum() + 0.5 * (v * v).sum()
    gx, gv = torch.autograd.grad(value, (x0, v0))
    return {"value": float(value), "dx": _host(gx), "dv": _host(gv)}


def _exact_fire(w, case, k):
    """FIRE as the reference's minimizerVertexLoop, per system."""
    batch = case["kind"] == "batch_fire"
    dt = k["dt"] * torch.ones(w.S, dtype=torch.float64, device=w.dev)
    if batch:  # the time step is given in mean ring sizes
        of_system = w.system[w.first == torch.arange(w.nv, device=w.dev)]
        size = torch.zeros_like(dt).index_add(0, of_system, w.a0) / torch.bincount(of_system, minlength=w.S)
        dt = dt * 2.0 * torch.sqrt(size / math.pi)
    a_start, f_dec, f_inc, f_a = FIRE
    x, v = w.x, torch.zeros_like(w.x)
    dt_max, alpha, n = 10.0 * dt, torch.full_like(dt, 0.2), torch.zeros_like(dt)
    f, e = w.force(x, energy=True)
    for _ in range(case["steps"]):
        power = w.per_system((v * f).sum(1))
        up = power > 0
        n = torch.where(up, n + 1, torch.zeros_like(n))
        grow = up & (n > FIRE_MIN_STEP)
        dt = torch.where(grow, torch.minimum(dt * f_inc, dt_max), dt)
        alpha = torch.where(grow, alpha * f_a, alpha)
        dt = torch.where(up, dt, torch.maximum(dt * f_dec, dt_max / 10))
        alpha = torch.where(up, alpha, torch.full_like(alpha, a_start))
        back, step = (~up)[w.system][:, None], dt[w.system][:, None]
        x = torch.where(back, x - 0.5 * step * v, x)
        v = torch.where(back, torch.zeros_like(v), v) + 0.5 * step * f
        ratio = torch.sqrt(w.per_system((v * v).sum(1)) / w.per_system((f * f).sum(1)))
        mix = alpha[w.system][:, None]
        v = (1 - mix) * v + mix * f * ratio[w.system][:, None]
        x = x + step * v
        f, e = w.force(x, energy=True)
        v = v + 0.5 * step * f
    if batch:
        return {"pos": _host(x), "vel": _host(v), "energies": _host(e), "iterations": None}
    return {"pos": _host(x), "vel": _host(v), "energy": float(e.sum() + 0.5 * (v * v).sum()), "iterations": None}


def _exact_rigid(w, case, seed):
    k, dt = w.k, w.k["dt"]
    noise = math.sqrt(2.0 * k["T"] * k["gamma"] / dt)
    is_first = w.first == torch.arange(w.nv, device=w.dev)
    nvr = w.nvr[:, None]
    c = torch.zeros(w.np, 2, dtype=torch.float64, device=w.dev)
    sums = lambda values: torch.zeros((w.np,) + values.shape[1:], dtype=torch.float64, device=w.dev).index_add(0, w.ring, values)  # noqa: E731
    c = w.x[is_first] + sums(w.x - w.x[w.first]) / nvr
    rel = w.x - c[w.ring]
    v, spin = w.v[is_first], torch.zeros(w.np, dtype=torch.float64, device=w.dev)

    def ring_force(x):
        y = x.detach().requires_grad_(True)
        e = w.pairs_energy(y, torch.zeros(w.S, dtype=torch.float64, device=w.dev))
        f = -torch.autograd.grad(e.sum(), y)[0]
        r = x - c[w.ring]
        return sums(f), sums(r[:, 0] * f[:, 1] - r[:, 1] * f[:, 0]) / sums((r * r).sum(1))

    f, turn = ring_force(w.x)
    for n in range(case["steps"]):
        v, spin = v + 0.5 * dt * f, spin + 0.5 * dt * turn
        c = c + dt * v
        cs, sn = torch.cos(dt * spin)[w.ring], torch.sin(dt * spin)[w.ring]
        rel = torch.stack([rel[:, 0] * cs - rel[:, 1] * sn, rel[:, 0] * sn + rel[:, 1] * cs], dim=1)
        x = c[w.ring] + rel
        f, turn = ring_force(x)
        f = f + noise * torch.as_tensor(_normals(1234 + seed % 1000, 2 * n, w.np), device=w.dev) - k["gamma"] * v
        v, spin = v + 0.5 * dt * f, spin + 0.5 * dt * turn
    return {"pos": _host(x), "vel": _host(v), "spin": _host(spin)}
