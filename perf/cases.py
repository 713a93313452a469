"""The performance cases of the kDOP collision library.

A case is one collision step as a user's program makes it: new positions in
(rigid poses, world vertices or a deformation phase), the trees refitted, the
mesh pairs traversed, contacts generated, and the results read in a
reproducible order -- through the Python binding and the C ABI it wraps.  The
meshes are the seeded tetrahedral lattices of kdop_b200.scenes, the shapes and
sizes the benchmark configurations and their neighbourhood: one pair to
thousands of bodies, a few hundred tets to tens of millions, every slab count.

  kind "step"    refit + traversal + contacts of a list of mesh pairs
  kind "dropin"  the same for one pair with host arrays in and out and the
                 refitted trees read back (what the C++ tag does per step)
  kind "diff"    contact depths differentiated with respect to the vertices
  kind "pile"    many small bodies: broad phase, then a step, then reduction
  kind "rows"    reduction of contact rows that a caller already holds
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "bvh-tvcg18_b200"))

import kdop_b200 as kd  # noqa: E402
from kdop_b200 import autograd, scenes  # noqa: E402


def _step(name, pairs, cells, K, pose, *, cells_lo=0, refit="pose", memory="device", graph=False, surface_filter=True,
          out="contacts"):
    case = {"kind": "step", "pairs": pairs, "cells": cells, "cells_lo": cells_lo or cells, "K": K, "pose": pose,
            "refit": refit, "memory": memory, "graph": graph, "surface_filter": surface_filter, "out": out}
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest call: two bodies of 384 tets that touch, poses from the host's integrator
        _step("touch_tiny", 1, 4, 14, "touch", memory="host"),
        # one ordinary pair, deep overlap, the sorted candidate pairs as the result (benchmark configuration 1)
        _step("pair_small", 1, 10, 14, "overlap", memory="host", out="candidates"),
        # the C++ drop-in's step: two 24,576-tet bodies, K = 8, positions up, trees and contacts back to the host
        {"name": "pair_dropin", "kind": "dropin", "cells": 16, "K": 8},
        # one huge pair with simulated vertices already on the device (configuration 2: 2 x 1.57 M tets)
        _step("pair_large", 1, 64, 26, "half", refit="vertices"),
        # the headline: 512 uneven pairs of 1 k to 200 k tets in one captured step (configuration 3)
        _step("batch_uneven", 512, 32, 14, "overlap", cells_lo=6, graph=True),
        # a few small uneven pairs of soft bodies uploaded by the host, all overlapping tet pairs wanted
        _step("batch_upload", 24, 7, 20, "overlap", cells_lo=2, refit="vertices", memory="host", surface_filter=False,
              out="candidates"),
        # 64 deforming, moving pairs of 384 k tets in one captured step (configuration 4)
        _step("deform_batch", 64, 40, 18, "touch", refit="deform", graph=True),
        # 256 resting contacts of 48 k-tet bodies, reduced to the solver's contact list (configuration 5)
        _step("touch_batch", 256, 20, 14, "touch", graph=True, out="reduced"),
        # an optimisation step: gradients of all contact depths back to the vertices (configuration 5's use)
        {"name": "diff_batch", "kind": "diff", "pairs": 64, "cells": 20, "K": 14},
        # the same for one small pair of odd size
        {"name": "diff_pair", "kind": "diff", "pairs": 1, "cells": 9, "K": 12},
        # a pile of many small bodies through the whole collision pipeline
        {"name": "pile", "kind": "pile", "bodies": 1500, "cells": 3, "K": 18},
        # a solver's own contact list reduced on the device
        {"name": "rows", "kind": "rows", "rows": 700001, "bodies": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges; single-pair meshes up to 100 k tets, batches up to about 6 M."""
    K = rng.choice((6, 8, 12, 14, 18, 20, 26))
    kind = rng.choice(("step", "step", "step", "step", "dropin", "diff", "pile", "rows"))
    if kind == "dropin":
        return {"kind": kind, "cells": _log_int(rng, 3, 24), "K": K}
    if kind == "diff":
        pairs = _log_int(rng, 1, 80)
        return {"kind": kind, "pairs": pairs, "cells": _log_int(rng, 3, 20 if pairs > 8 else 28), "K": K}
    if kind == "pile":
        return {"kind": kind, "bodies": _log_int(rng, 40, 3000), "cells": rng.randint(1, 4), "K": K}
    if kind == "rows":
        return {"kind": kind, "rows": _log_int(rng, 100, 2000000), "bodies": _log_int(rng, 4, 4000)}
    pairs = _log_int(rng, 1, 200)
    cells = _log_int(rng, 3, min(36, int((6e6 / (12 * pairs)) ** (1 / 3))))
    pose = rng.choice(("overlap", "touch"))
    refit = rng.choice(("pose", "vertices", "deform") if pose == "touch" else ("pose", "vertices"))
    everything = pairs * cells ** 3 <= 20000 and rng.random() < 0.3
    return _step("", pairs, cells, K, pose, cells_lo=max(2, cells // rng.randint(1, 4)) if pose == "overlap" else cells,
                 refit=refit, memory=rng.choice(("host", "device")), graph=rng.random() < 0.5,
                 surface_filter=not everything,
                 out="candidates" if everything or pairs * cells ** 3 <= 20000 and rng.random() < 0.3 else
                 rng.choice(("contacts", "reduced")))


# ---- inputs ---------------------------------------------------------------------

def _half_overlap(n, K, seed):
    """Two jittered n^3-cell lattices, B moved by half a side and turned by at most 10 degrees."""
    rng = np.random.default_rng(seed)
    meshes = [scenes.lattice(n, 0.2, rng) for _ in range(2)]
    quat = np.array([[1, 0, 0, 0], [1, 0, 0, 0]], np.float32)
    pos = np.zeros((2, 3), np.float32)
    quat[1] = scenes.axis_angle_quaternion(rng.normal(size=3), math.radians(10.0) * rng.uniform(0.0, 1.0))
    pos[1] = (n / 2.0, 0.0, 0.0)
    return scenes.Scene(f"2 x {n}^3 cells", K, meshes, quat, pos, np.array([[0, 1]], np.uint32))


def _pile(bodies, n_max, K, seed):
    """Bodies of 1 to n_max cells a side, each turned by up to 5 degrees, on a grid close enough to touch."""
    rng = np.random.default_rng(seed)
    sizes = rng.integers(1, n_max + 1, bodies)
    meshes = [scenes.lattice(int(n), 0.1, rng) for n in sizes]
    side = int(math.ceil(bodies ** (1 / 3)))
    cell = np.stack(np.unravel_index(np.arange(bodies), (side, side, side)), axis=1)
    pos = (cell * (0.9 * n_max) + rng.uniform(-0.1, 0.1, (bodies, 3))).astype(np.float32)
    quat = np.stack([scenes.axis_angle_quaternion(rng.normal(size=3), math.radians(5.0) * rng.uniform(-1.0, 1.0))
                     for _ in range(bodies)])
    return scenes.Scene(f"pile of {bodies}", K, meshes, quat, pos, np.zeros((0, 2), np.uint32))


def _scene(case, seed):
    K = case["K"]
    if case["kind"] == "pile":
        return _pile(case["bodies"], case["cells"], K, seed)
    if case["kind"] == "dropin":
        return scenes.touching_pair(case["cells"], seed, K, 0.1)
    if case["kind"] == "diff" or case["pose"] == "touch":
        return scenes.config5(case["pairs"], case["cells"], seed, K)
    if case["pose"] == "half":
        return _half_overlap(case["cells"], K, seed)
    return scenes.config3(case["pairs"], seed, 6 * (case["cells_lo"] - 0.4) ** 3, 6 * (case["cells"] + 0.4) ** 3,
                          0.15, K)


def _world(sc):
    """World positions of every mesh (the user's own simulated vertices), float32."""
    parts = []
    for m, q, p in zip(sc.meshes, sc.quat.astype(np.float64), sc.pos.astype(np.float64)):
        r = m.xyz.astype(np.float64)
        t = 2.0 * np.cross(q[1:], r)
        parts.append(r + q[0] * t + np.cross(q[1:], t) + p)
    return np.ascontiguousarray(np.concatenate(parts), np.float32)


def _rows(n, bodies, seed):
    """Contact rows of a touching scene: points in a box, axis-like normals, one row in four reported twice (by the
    neighbouring tet), some of those with a depth that differs in the last bits."""
    rng = np.random.default_rng(seed)
    base = n - n // 4
    p = rng.uniform(-20.0, 20.0, (base, 3)).astype(np.float32)
    nrm = rng.normal(size=(base, 3))
    nrm = (nrm / np.linalg.norm(nrm, axis=1, keepdims=True)).astype(np.float32)
    depth = rng.uniform(-0.5, 0.0, base).astype(np.float32)
    pair = np.sort(rng.integers(0, bodies, (base, 2)), axis=1).astype(np.uint32)
    twice = rng.integers(0, base, n - base)
    order = rng.permutation(n)
    again = depth[twice] + np.float32(2.0 ** -22) * rng.integers(0, 2, n - base).astype(np.float32)
    out = np.zeros((n, 8), np.float32)
    out[:, 0:3] = np.concatenate([p, p[twice]])[order]
    out[:, 3:6] = np.concatenate([nrm, nrm[twice]])[order]
    out[:, 6] = np.concatenate([depth, again])[order]
    out[:, 7] = np.arange(n, dtype=np.uint32).view(np.float32)
    return out, np.concatenate([pair, pair[twice]])[order]


def _capacity(case):
    """(candidate rows, contact rows) a program of this case keeps room for."""
    if case["kind"] == "pile":
        return 0, 220 * case["bodies"] * case["cells"] + 4096
    hi, pairs = case["cells"], case.get("pairs", 1)
    lo = case.get("cells_lo", hi)
    face = hi ** 2 if lo == hi else (hi ** 2 - lo ** 2) / (2 * math.log(hi / lo))  # mean of log-uniform sizes
    cube = hi ** 3 if lo == hi else (hi ** 3 - lo ** 3) / (3 * math.log(hi / lo))
    face, cube = pairs * face + 2 * hi ** 2, pairs * cube + 2 * hi ** 3
    touch = case.get("pose", "touch") == "touch"
    rows = 48 * face + 1000 * pairs if case.get("surface_filter", True) else 160 * cube + 1000 * pairs
    return int(rows) + 4096, int((64 if touch else 12) * face) + 4096


def prepare(case, seed):
    ctx = kd.Context(0)
    if case["kind"] == "rows":
        rows, bodies = _rows(case["rows"], case["bodies"], seed)
        n = case["rows"]
        return {"case": case, "ctx": ctx, "rows": torch.from_numpy(rows).cuda(),
                "bodies": torch.from_numpy(bodies.view(np.int32)).cuda(),
                "out": torch.zeros((n, 8), dtype=torch.float32, device="cuda"),
                "out_bodies": torch.zeros((n, 2), dtype=torch.int32, device="cuda")}
    sc = _scene(case, seed)
    scene = kd.DeviceScene(ctx, sc.K, sc.meshes)
    st = {"case": case, "ctx": ctx, "scene": scene, "pairs": sc.pairs}
    device = case.get("memory") == "device"
    put = (lambda a: torch.from_numpy(a).cuda()) if device else (lambda a: torch.from_numpy(a).pin_memory())
    kind, mode = case["kind"], case.get("refit", "pose")
    if kind == "diff":
        st["xyz"] = torch.from_numpy(_world(sc)).cuda().requires_grad_(True)
        scene.set_vertices(st["xyz"].detach())
        scene.refit(kd.REFIT_VERTICES)
    elif kind == "dropin":
        st["xyz"] = _world(sc)
        scene.set_vertices(st["xyz"])
        scene.refit(kd.REFIT_VERTICES)
    elif mode == "vertices":
        st["xyz"] = put(_world(sc))
        scene.set_vertices(st["xyz"])
        scene.refit(kd.REFIT_VERTICES)
    else:
        st["quat"], st["pos"] = put(sc.quat), put(sc.pos)
        st["phase"] = float(np.random.default_rng(seed).uniform(0.0, 2.0 * math.pi))
        scene.set_poses(st["quat"], st["pos"])
        if mode == "deform":
            scene.set_deformation(0.1, 2.0 * math.pi / case["cells"], st["phase"])
        scene.refit(kd.REFIT_DEFORM if mode == "deform" else kd.REFIT_POSE)
    # the buffers a program's first step has grown
    if kind == "pile":
        st["pairs"] = scene.broad_phase()
    st["opts"] = None if case.get("surface_filter", True) else scene.opts(surface_filter=0)
    s = scene.traverse_sync(st["pairs"], st["opts"], contacts=True)
    scene.reserve(int(1.25 * s.n_candidates) + 1024, int(1.25 * s.n_contacts) + 1024)
    # the program's own result buffers, of one size for all its steps: device memory, or pinned host memory where the
    # results go back to the host
    rows, contacts = _capacity(case)
    where = {"pin_memory": True} if kind in ("dropin", "pile") else {"device": "cuda"}
    if case.get("out") == "candidates":
        st["out"] = torch.zeros((rows, 3), dtype=torch.int32, pin_memory=True)
    elif kind != "diff":
        st["out"] = torch.zeros((contacts, 8), dtype=torch.float32, **where)
        st["out_bodies"] = torch.zeros((contacts, 2), dtype=torch.int32, **where)
    if kind == "pile":
        st["out_pairs"] = torch.zeros((64 * case["bodies"] + 1024, 2), dtype=torch.int32, pin_memory=True)
    if kind == "step":
        if case["graph"]:
            scene.graph_capture(st["pairs"], {"vertices": kd.REFIT_VERTICES, "pose": kd.REFIT_POSE,
                                              "deform": kd.REFIT_DEFORM}[mode], st["opts"])
    ctx.synchronize()
    return st


# ---- one pass ---------------------------------------------------------------------
# The result buffers are returned whole: rows past the counts stay as they were.

def _fields(rows):
    """Contact rows (n, 8) as the fields they hold."""
    return {"p": rows[:, 0:3], "n": rows[:, 3:6], "depth": rows[:, 6], "cand": rows[:, 7].view(torch.int32)}


def _reduce(st):
    """kdop_reduce_contacts into the program's buffers."""
    scene, n = st["scene"], ctypes.c_int64()
    rc = scene.lib.kdop_reduce_contacts(scene.h, st["out"].data_ptr(), st["out_bodies"].data_ptr(),
                                        st["out"].shape[0], ctypes.byref(n))
    scene.ctx._check(rc, "kdop_reduce_contacts")
    return {"kept": n.value, "rows": st["out"][:, :7], "bodies": st["out_bodies"]}


def _run_step(st):
    case, scene = st["case"], st["scene"]
    mode = case["refit"]
    if mode == "vertices":
        scene.set_vertices(st["xyz"])
    else:
        scene.set_poses(st["quat"], st["pos"])
        if mode == "deform":
            scene.set_deformation(0.1, 2.0 * math.pi / case["cells"], st["phase"])
    if case["graph"]:
        scene.graph_launch()
    else:
        scene.refit({"vertices": kd.REFIT_VERTICES, "pose": kd.REFIT_POSE, "deform": kd.REFIT_DEFORM}[mode])
        scene.traverse(st["pairs"], st["opts"])
        if case["out"] != "candidates":
            scene.contacts()
    s = scene.stats()
    out = {"tests": int(s.n_tests), "candidates": int(s.n_candidates)}
    if case["out"] == "reduced":
        return dict(out, **_reduce(st))
    scene.sort_results()
    if case["out"] == "contacts":
        return dict(out, contacts=scene.read_contacts_into(st["out"]), **_fields(st["out"]))
    n = ctypes.c_int64()
    rc = scene.lib.kdop_read_candidates(scene.h, st["out"].data_ptr(), st["out"].shape[0], ctypes.byref(n))
    scene.ctx._check(rc, "kdop_read_candidates")
    return dict(out, rows=st["out"])


def _run_dropin(st):
    scene = st["scene"]
    scene.set_vertices(st["xyz"])
    scene.refit(kd.REFIT_VERTICES)
    trees = [scene.read_tree(m) for m in range(2)]
    s = scene.traverse_sync(st["pairs"], contacts=True)
    scene.sort_results()
    n = scene.read_contacts_into(st["out"])
    return {"vol": [t[0] for t in trees], "tet": [t[1] for t in trees], "tests": int(s.n_tests), "contacts": n,
            **_fields(st["out"])}


def _run_diff(st):
    depth, normal = autograd.contact_geometry(st["xyz"], st["scene"], st["pairs"])
    loss = (depth * depth).sum()
    grad, = torch.autograd.grad(loss, st["xyz"])
    return {"loss": loss.detach(), "contacts": int(depth.shape[0]), "grad": grad}


def _run_pile(st):
    scene = st["scene"]
    scene.set_poses(st["quat"], st["pos"])
    scene.refit(kd.REFIT_POSE)
    n = ctypes.c_int64()
    rc = scene.lib.kdop_broad_phase(scene.h, None, kd.HOST, st["out_pairs"].data_ptr(), st["out_pairs"].shape[0],
                                    ctypes.byref(n))
    scene.ctx._check(rc, "kdop_broad_phase")
    s = scene.traverse_sync(st["out_pairs"][:n.value].numpy().view(np.uint32), contacts=True)
    return {"pairs": st["out_pairs"], "found": n.value, "tests": int(s.n_tests), **_reduce(st)}


def _run_rows(st):
    n = ctypes.c_int64()
    rc = st["ctx"].lib.kdop_reduce_contact_rows(st["ctx"].h, st["rows"].data_ptr(), st["bodies"].data_ptr(),
                                                st["rows"].shape[0], st["out"].data_ptr(),
                                                st["out_bodies"].data_ptr(), st["out"].shape[0], ctypes.byref(n))
    st["ctx"]._check(rc, "kdop_reduce_contact_rows")
    return {"kept": n.value, "rows": st["out"][:, :7], "bodies": st["out_bodies"]}


def run(state):
    return {"step": _run_step, "dropin": _run_dropin, "diff": _run_diff, "pile": _run_pile,
            "rows": _run_rows}[state["case"]["kind"]](state)


# ---- what a pass cannot do without ------------------------------------------------

def work(case):
    """Bytes: positions and tets read once, every node's slabs written once (the updated trees), contact rows in and
    out.  Operations: the projections of four vertices on K/2 directions per tet and the unions above them."""
    kind = case["kind"]
    if kind == "rows":
        n = case["rows"]
        return {"bytes": 40.0 * n + 40.0 * 0.75 * n, "flops": 9.0 * n * max(1.0, math.log2(n))}
    if kind == "pile":
        tets = case["bodies"] * sum(6.0 * n ** 3 for n in range(1, case["cells"] + 1)) / case["cells"]
    else:
        lo, hi = 6.0 * case.get("cells_lo", case["cells"]) ** 3, 6.0 * case["cells"] ** 3
        mean = hi if hi <= 1.01 * lo else (hi - lo) / math.log(hi / lo)  # log-uniform sizes
        tets = 2.0 * case.get("pairs", 1) * mean
    K = case["K"]
    return {"bytes": tets * (16.0 + 12.0 / 5.0 + 2 * 4.0 * K), "flops": tets * (4 * (K // 2) * 5.0 + 4.0 * K)}


# ---- 64-bit values ----------------------------------------------------------------

def _directions(K):
    """Unit slab directions in the order of the K-DOP tables: axes, corners, edges."""
    axes = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]
    corners = [(1, 1, 1), (1, 1, -1), (1, -1, 1), (1, -1, -1)]
    edges = [(1, 1, 0), (1, -1, 0), (1, 0, 1), (0, 1, 1), (-1, 0, 1), (0, -1, 1)]
    d = np.array({6: axes, 8: corners, 12: edges, 14: axes + corners, 18: axes + edges, 20: corners + edges,
                  26: axes + corners + edges}[K], np.float64)
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _leaf_order(mesh):
    """Tets by Morton code of their rest centroid: 21 bits an axis, one integer scale, x in the lowest bit."""
    v = mesh.xyz[mesh.tets.astype(np.int64)]
    c = (0.25 * (((v[:, 0] + v[:, 1]) + v[:, 2]) + v[:, 3]).astype(np.float64)).astype(np.float32)
    lo = c.min(axis=0)
    hi = np.maximum(c.max(axis=0), np.finfo(np.float32).tiny)
    scale = np.float32(int(np.min(np.float32((1 << 21) - 1) / (hi - lo))))
    q = ((c - lo) * scale).astype(np.int64).astype(np.uint64)
    code = np.zeros(len(c), np.uint64)
    for bit in range(21):
        for axis in range(3):
            code |= ((q[:, axis] >> np.uint64(bit)) & np.uint64(1)) << np.uint64(3 * bit + axis)
    return np.argsort(code, kind="stable")


def _exact_tree(mesh, world, K):
    """Slabs of every node in preorder: index-median splits of the leaf order down to one tet."""
    n = mesh.n_tets
    order = _leaf_order(mesh)
    proj = world.astype(np.float64)[mesh.tets[order].astype(np.int64)] @ _directions(K).T
    lo, hi = proj.min(axis=1), proj.max(axis=1)
    vol = np.zeros((2 * n - 1, K))
    first, size, at = np.array([0]), np.array([n]), np.array([0])
    while len(first):  # one level at a time: the tet range and the preorder index of its nodes
        cut = np.stack([first, first + size], axis=1).ravel()
        pad = lambda a, v: np.concatenate([a, np.full((1, a.shape[1]), v)])  # noqa: E731
        vol[at, 0::2] = np.minimum.reduceat(pad(lo, np.inf), cut)[0::2]
        vol[at, 1::2] = np.maximum.reduceat(pad(hi, -np.inf), cut)[0::2]
        first, size, at = first[size > 1], size[size > 1], at[size > 1]
        left = size - size // 2
        first = np.stack([first, first + left], axis=1).ravel()
        at = np.stack([at + 1, at + 2 * left], axis=1).ravel()
        size = np.stack([left, size - left], axis=1).ravel()
    return vol


def _exact_dropin(case, seed):
    sc = _scene(case, seed)
    xyz = np.split(_world(sc), [sc.meshes[0].n_verts])
    return {"vol": [_exact_tree(m, x, case["K"]) for m, x in zip(sc.meshes, xyz)], "tet": [None, None],
            "tests": None, "contacts": None, "p": None, "n": None, "depth": None, "cand": None}


def _exact_rows(case, seed):
    rows, bodies = _rows(case["rows"], case["bodies"], seed)
    key = [rows[:, c].astype(np.float64) for c in (6, 5, 3, 4, 2, 0, 1)] + [bodies[:, 1], bodies[:, 0]]
    order = np.lexsort(key)
    rows, bodies = rows[order].astype(np.float64), bodies[order]
    # a row is dropped when the row before it is the same report (its depth may differ in the last bits)
    new = np.ones(len(rows), bool)
    new[1:] = np.any(rows[1:, :6] != rows[:-1, :6], axis=1) | np.any(bodies[1:] != bodies[:-1], axis=1)
    out = np.zeros((len(rows), 7))
    out[:new.sum()] = rows[new, :7]
    return {"kept": None, "rows": torch.from_numpy(out), "bodies": None}


def exact(case, seed):
    """The refitted trees and the reduced rows in 64 bits.  Contact rows and their gradients have no such value: which
    of the 56 points of a tet pair lie inside is decided by single-precision rounding (an edge/plane crossing lies on
    the plane it is tested against), so a 64-bit run keeps other points.  Candidates and counts are whole numbers."""
    if case["kind"] == "rows":
        return _exact_rows(case, seed)
    return _exact_dropin(case, seed) if case["kind"] == "dropin" else None
