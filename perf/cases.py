"""Performance cases of the collision path: what a user's program calls, at the
sizes and in the settings it meets.

A case is a dict of plain values:

``path``    the entry points of one pass
            ``step``        DevicePipeline.run: boxes, pairs and contacts of one
                            resident scene, the call of a simulation's time step
            ``classes``     GenerateAABB, detectPossibleCollisions and DoNarrowphase
                            one after the other, as code written for the
                            reference's three classes calls them
            ``broadphase``  GenerateAABB and detectPossibleCollisions only
            ``batch``       BatchPipeline.run: many scenes of uneven size at once
            ``served``      perturb_many and ScenesPipeline.run: a server's pass
                            over scenes that live in their own allocations
            ``stepping``    perturb_ and DevicePipeline.run with candidate lists
                            kept from step to step (set_incremental)
            ``host``        HostSession.run: host arrays in, host arrays out
``scene``   ``spheres`` (one size range, cube), ``mixed`` (spheres, boxes,
            ellipsoids and cylinders), ``clustered`` (spheres in Gaussian
            clusters: cells from empty to thousands of boxes)
``n``       shapes (``batch`` and ``served``: of the largest scene)
``crowding`` box pairs per body: 0.026 is the 1M-shape workload's gas of small
            bodies, a settled granular heap has a few
``precision`` narrowphase mode: exact, fp64 or mixed

Passes whose result the library allocates (``classes``, ``broadphase``) take
one fixed scene with its bodies in an order drawn from the seed; the others
return the pipeline's own buffers, zero behind the valid rows, and the counts.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "collision-detection_b200"))

import collide_b200 as cb  # noqa: E402
from collide_b200 import scenes, serving  # noqa: E402

GRID = (16, 16, 16)   # the reference's default bins per axis


def _case(name, path, scene, n, crowding=0.026, precision="exact", count=1):
    c = dict(path=path, scene=scene, n=int(n), crowding=float(crowding), precision=precision, count=int(count))
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small heap in a control or planning loop: the call's latency is all that counts
        _case("step_mixed_1k", "step", "mixed", 1000, 2.0),
        # the plain-method workload, 16,384 equal-ish spheres with a contact here and there
        _case("step_spheres_16k", "step", "spheres", 16384, 0.04),
        # an ordinary gas of mixed convex bodies, ragged size
        _case("step_mixed_130k", "step", "mixed", 130003),
        # the headline workload
        _case("step_mixed_1m", "step", "mixed", 1 << 20),
        # granular heaps: several candidate pairs per body, most of them contacts to refine
        _case("step_heap_50k", "step", "mixed", 50021, 4.0),
        _case("step_heap_200k_fp64", "step", "mixed", 200003, 3.0, "fp64"),
        # a program ported from the reference: its three calls in turn, on its timing test's distribution
        _case("classes_spheres_20k", "classes", "spheres", 20011, 0.8),
        # astrophysics-like density contrast, broadphase alone: hundreds of pairs per body
        _case("broadphase_clustered_4m", "broadphase", "clustered", 1 << 22),
        # parameter studies: many independent scenes of log-uniform size in one pass
        _case("batch_64", "batch", "mixed", 100000, count=64),
        # a server's pass: every resident scene takes its time step, then all are collided
        _case("served_16", "served", "mixed", 200000, count=16),
        # a simulation whose bodies move a little per step
        _case("stepping_mixed_500k", "stepping", "mixed", 500009),
        # scene data on the host, as a CPU solver has it
        _case("host_mixed_60k", "host", "mixed", 60013, 0.5),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    path = rng.choice(("step", "step", "step", "step", "classes", "broadphase", "batch", "served", "stepping", "host"))
    crowding = round(math.exp(rng.uniform(math.log(0.02), math.log(4.0))), 4)
    if path == "step":
        n = size(500, 1 << 20)
        crowding = min(crowding, 4.0 * 50000 / max(n, 50000))
        return _case(None, path, rng.choice(("spheres", "mixed", "mixed")), n, crowding,
                     rng.choice(("exact", "exact", "fp64", "mixed")))
    if path == "classes":
        return _case(None, path, "spheres", size(1000, 130000), min(crowding, 1.0))
    if path == "broadphase":
        return _case(None, path, rng.choice(("clustered", "spheres")), size(20000, 1 << 22), min(crowding, 1.0))
    if path == "batch":
        return _case(None, path, "mixed", size(4000, 100000), min(crowding, 0.2), count=rng.randint(3, 64))
    if path == "served":
        return _case(None, path, "mixed", size(4000, 200000), min(crowding, 0.1), count=rng.randint(2, 16))
    if path == "stepping":
        return _case(None, path, "mixed", size(20000, 500009), min(crowding, 0.1))
    return _case(None, path, "mixed", size(2000, 130000), min(crowding, 0.5))


# ---------------------------------------------------------------- scenes
def _volume(n, crowding, mean_cube):
    """Volume in which n boxes make `crowding` overlapping pairs per box:
    n / (2 V) times the mean volume in which two boxes overlap."""
    return n * mean_cube / (2.0 * crowding)


def _scene(kind, n, crowding, seed):
    if kind == "clustered":
        return scenes.clustered_spheres(n, seed=seed)
    if kind == "spheres":  # radii U[0.002, 0.006]: boxes of mean edge 0.008
        edge = _volume(n, crowding, 0.0161 ** 3) ** (1.0 / 3.0)
        return scenes.spheres_uniform(n, seed=seed, hi=edge)
    # mixed: half extents U[0.001, 0.004] turned at random; a flat slab for the gas, a squat heap when crowded
    v = _volume(n, crowding, 0.0135 ** 3)
    flat = 20.0 if crowding < 0.1 else 2.0
    z = (v / flat ** 2) ** (1.0 / 3.0)
    return scenes.mixed_slab(n, seed=seed, extent=(flat * z, flat * z, z))


def _one(case, seed):
    if case["path"] not in ("classes", "broadphase"):
        return _scene(case["scene"], case["n"], case["crowding"], seed)
    s = _scene(case["scene"], case["n"], case["crowding"], 5)
    order = np.random.Generator(np.random.PCG64(seed)).permutation(s.n)
    s.B, s.pos = np.ascontiguousarray(s.B[order]), np.ascontiguousarray(s.pos[order])  # spheres: all else is alike
    return s


def _many(case, seed):
    return [_scene("mixed", k, case["crowding"], seed * 1009 + i) for i, k in enumerate(_sizes(case))]


def _sizes(case):
    """Sizes of the scenes of a batch or a pass: they belong to the case, positions and shapes to the seed."""
    rng = np.random.Generator(np.random.PCG64(7))
    k = np.exp(rng.uniform(np.log(min(1000, case["n"])), np.log(case["n"]), case["count"])).round().astype(int)
    k[0] = case["n"]
    return k.tolist()


def _shapes(case):
    return sum(_sizes(case)) if case["path"] in ("batch", "served") else case["n"]


# ---------------------------------------------------------------- passes
def _context(case):
    ctx = cb.Context()
    ctx.set_narrowphase_precision(case["precision"])
    return ctx


def _cleared(p):
    for t in (p.pairs, p.norm, p.cpta, p.cptb, p.depth, p.bids):
        t.zero_()
    return p


def prepare(case, seed):
    path, ctx = case["path"], _context(case)
    if path == "batch":
        db = cb.DeviceBatch(_many(case, seed))
        return dict(path=path, p=_cleared(cb.BatchPipeline(db, GRID, ctx=ctx, pairs_cap=_room(case))))
    if path == "served":
        p, held = cb.ScenesPipeline(ctx, GRID, pairs_cap=_room(case)), [cb.DeviceScene(s) for s in _many(case, seed)]
        p.run(held)  # a server sizes its buffers before it takes queries
        return dict(path=path, p=_cleared(p), scenes=held, ctx=ctx, t=0)
    sc = _one(case, seed)
    if path == "host":
        return dict(path=path, p=_cleared(cb.HostSession(sc, GRID, ctx=ctx, pairs_cap=_room(case))))
    ds = cb.DeviceScene(sc)
    if path in ("step", "stepping"):
        if path == "stepping":
            ctx.set_incremental(True, 2.0)
        p = _cleared(cb.DevicePipeline(ds, GRID, ctx=ctx, pairs_cap=_room(case)))
        return dict(path=path, p=p, ds=ds, ctx=ctx, t=0)
    aabb = torch.zeros((2 * sc.n, 3), dtype=torch.float32, device=ds.T.device)
    return dict(path=path, ds=ds, aabb=aabb, gen=cb.AABBGenerator(ctx), bp=cb.Broadphase(ctx), np=cb.Narrowphase(ctx))


def _room(case):
    """Room for the pairs, as a program that knows its scene allots it."""
    return int(_shapes(case) * max(0.25, 1.5 * case["crowding"])) + 1024


def _results(p):
    out = dict(pairs=p.pairs, norm=p.norm, cpta=p.cpta, cptb=p.cptb, depth=p.depth, bids=p.bids, n_pairs=p.n_pairs,
               n_contacts=p.n_contacts)
    return out if p.aabb is None else dict(out, aabb=p.aabb)


def run(state):
    path = state["path"]
    if path in ("classes", "broadphase"):
        ds = state["ds"]
        aabb = state["gen"].GenerateAABB(ds.T, ds.A, ds.B, ds.C, ds.R, ds.ID, ds.pos, ds.rot, state["aabb"])
        pairs = state["bp"].detectPossibleCollisions(aabb)
        if path == "broadphase":
            return dict(aabb=aabb, pairs=pairs)
        norm, cpta, cptb, depth, bids, _ = state["np"].DoNarrowphase(ds.T, ds.A, ds.B, ds.C, ds.R, ds.ID, ds.active,
                                                                     ds.pos, ds.rot, pairs)
        return dict(pairs=pairs, norm=norm, cpta=cpta, cptb=cptb, depth=depth, bids=bids, aabb=aabb)
    p = state["p"]
    if path == "served":
        state["t"] += 1
        serving.perturb_many(state["ctx"], [(s, state["t"] * 64 + i) for i, s in enumerate(state["scenes"])])
        p.run(state["scenes"])
        return dict(_results(p), scene_pairs=p.scene_pairs.astype(np.int64),
                    contact_offsets=p.contact_offsets.astype(np.int64))
    if path == "stepping":
        state["t"] += 1
        serving.perturb_(state["ctx"], state["ds"], state["t"])
        p.run()
        return dict(_results(p), pos=state["ds"].pos, rot=state["ds"].rot)
    p.run()
    if path == "batch":
        return dict(_results(p), scene_pairs=p.scene_pairs.astype(np.int64),
                    contact_offsets=p.contact_offsets.astype(np.int64))
    return _results(p)


def work(case):
    n = _shapes(case)
    # each shape and body read once (T, A, B, R, ID, position, rotation, flag), its box written once
    shape_in, box = 4 + 12 + 12 + 16 + 4 + 12 + 16, 24
    if case["scene"] == "clustered":  # pairs of the 64-cluster scene: 3.95e9 at 2^24 bodies, quadratic in n
        pairs = 3.95e9 * (n / 2.0 ** 24) ** 2
    else:
        pairs = n * case["crowding"]
    if case["path"] == "broadphase":
        return {"bytes": n * (shape_in + box) + 8 * pairs, "flops": 60.0 * n}
    moved = 2 * 28 * n if case["path"] in ("stepping", "served") else 0  # poses read and written by the update
    contacts = 0.35 * pairs
    refined = contacts * (0.0 if case["scene"] == "spheres" else 0.9)
    return {"bytes": n * (shape_in + 1 + box) + moved + 8 * pairs + 48 * contacts, "flops": 60.0 * n + 8800.0 * refined}


# ---------------------------------------------------------------- exact values
def _rows(q):
    w, x, y, z = (q[:, i] for i in range(4))
    return np.stack([np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)], 1),
                     np.stack([2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)], 1),
                     np.stack([2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1)], 1)


def _boxes(s):
    """Shifted boxes in 64 bits: one shape per body, no local offset or turn."""
    B, pos = s.B.astype(np.float64), s.pos.astype(np.float64)
    half = np.empty_like(B)
    sph = s.T == scenes.SPHERE
    half[sph] = B[sph, :1]
    rest = ~sph
    half[rest] = np.einsum("nij,nj->ni", np.abs(_rows(s.rot[rest].astype(np.float64))), B[rest])
    box = np.concatenate([pos - half, pos + half])
    return box + np.abs(box[: s.n].min(0))


def _sphere_contacts(s):
    """Contacts of a sphere scene in 64 bits, in the order of the pairs."""
    x, r = torch.from_numpy(s.pos).double(), torch.from_numpy(s.B[:, 0].copy()).double()
    ii, jj = [], []
    for i0 in range(0, s.n, 512):
        xi, ri = x[i0:i0 + 512], r[i0:i0 + 512]
        d2 = sum((x[None, i0:, d] - xi[:, None, d]) ** 2 for d in range(3))
        hit = torch.nonzero(d2 <= (ri[:, None] + r[None, i0:]) ** 2)
        hit = hit[hit[:, 1] > hit[:, 0]] + i0
        ii.append(hit[:, 0])
        jj.append(hit[:, 1])
    i, j = torch.cat(ii), torch.cat(jj)
    rel = x[j] - x[i]
    norm = rel / rel.norm(dim=1, keepdim=True)
    pa, pb = x[i] + r[i, None] * norm, x[j] - r[j, None] * norm
    return dict(norm=norm, cpta=pa, cptb=pb, depth=((pb - pa) * norm).sum(1))


def exact(case, seed):
    path = case["path"]
    if path in ("served", "stepping"):  # the poses are a random walk of the update's own single-precision arithmetic
        return None
    out = dict(pairs=None, norm=None, cpta=None, cptb=None, depth=None, bids=None)
    if path not in ("classes", "broadphase"):
        out.update(n_pairs=None, n_contacts=None)
    if path == "batch":
        per = [_boxes(s) for s in _many(case, seed)]
        half = [b.shape[0] // 2 for b in per]
        box = np.concatenate([b[:h] for b, h in zip(per, half)] + [b[h:] for b, h in zip(per, half)])
        return dict(out, aabb=box, scene_pairs=None, contact_offsets=None)
    if path == "host":
        return None
    s = _one(case, seed)
    if path == "broadphase":
        return dict(aabb=_boxes(s), pairs=None)
    # the contacts of the other shapes come from an iteration that stops at a portal, not from a formula
    if case["scene"] == "spheres" and case["n"] <= 32768:
        for k, v in _sphere_contacts(s).items():
            if path == "step":  # the whole buffer: zero behind the contacts
                full = torch.zeros((_room(case),) + tuple(v.shape[1:]), dtype=torch.float64)
                full[: v.shape[0]] = v
                v = full
            out[k] = v
    return dict(out, aabb=_boxes(s))
