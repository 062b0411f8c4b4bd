"""What this backend is timed on: the calls a fragment-reassembly program makes, from one pose's
verification to a collection's batched ladder, over generated fragments (synth).

A case names an operation and its sizes; the fragments, samples and poses come from the seed.

  verify      Context.verify: R 6's scores of one pose (a user placing a join by hand).
  stage2      Context.ladder_verify_batch on host buffers: the four rungs, R 6 and the verdict of
              every (pair, start); one pair is what match_pair asks, a pot what match_collection.
  resident    Batch.run + results on a batch kept on the device (a collection, run over and over).
  icp         Executor.icp_rung: one point-to-plane rung for a pair's starts.
  stage1      PairStage1.run: hypotheses, coarse scores, suppression, the point-to-point ladder.
  inside      Context.inside: parity and depth of surface samples in the other fragment.
  distance    Context.bounded_distance: samples against the other fragment's fracture faces.
  nearest     Cloud.nearest_below: bounded nearest neighbours of one sampled surface in another.
  preprocess  one fragment from its mesh: upload, face geometry, wall thickness, segmentation and
              breaklines (R 3.2-3.5; the breaklines of the generator's labels, so that their count
              does not hang on a vote).
  refine      R 9 of one join: both fracture clouds from the original meshes, then the two rungs.
  adjoint     Context.adjoint: objectives and twist gradients of an assembled pot's edges at many
              group poses (one evaluation of the joint refinement).
"""

from __future__ import annotations

import functools
import importlib
import math

import numpy as np
import torch

PACKAGE = "sherd-refit_b200"
sherd = importlib.import_module(PACKAGE)
preprocess = importlib.import_module(PACKAGE + ".preprocess")
refine = importlib.import_module(PACKAGE + ".refine")
stage1 = importlib.import_module(PACKAGE + ".stage1")
synth = importlib.import_module(PACKAGE + ".synth")
workload = importlib.import_module(PACKAGE + ".workload")


@functools.lru_cache(maxsize=1)
def context():
    """The process's one context, as a program holds it."""
    return sherd.Context(0)


def listed():
    return [
        # One candidate join checked at one pose: the smallest call of the matching path.
        {"name": "verify_pose", "op": "verify", "edges": 7.0},
        # match_pair's stage 2: the ten starts stage 1 leaves of one pair, host buffers.
        {"name": "stage2_pair", "op": "stage2", "edges": 7.0, "cells": 0, "starts": 10,
         "early": 0.0},
        # match_collection's stage 2 on one pot of 8 fragments: 28 pairs, 64 starts each.
        {"name": "stage2_pot", "op": "stage2", "edges": 6.5, "cells": 8, "starts": 64, "t": 12.0,
         "frac_per_t2": 150.0, "frac_max": 12000, "early": 0.0},
        # A collection of two walls, fracture clouds of 1k-60k points, resident on the device.
        {"name": "resident_collection", "op": "resident", "edges": 7.0, "cells": 6, "walls": 2,
         "starts": 128, "t": 10.0, "frac_per_t2": 900.0, "frac_max": 60000, "early": 0.0},
        # One executor rung at stage 2's sizes.
        {"name": "icp_rung", "op": "icp", "edges": 7.0, "starts": 10, "k": 0.2},
        # Stage 1 of one pair.
        {"name": "stage1_pair", "op": "stage1", "edges": 5.0},
        # R 8's question for one placed pair: 20 000 surface samples in the other mesh.
        {"name": "inside_samples", "op": "inside", "edges": 7.0, "n": 20000},
        # A full-resolution fracture surface measured against the other one, an odd count.
        {"name": "distance_samples", "op": "distance", "edges": 7.0, "n": 150001},
        # Dense surface against dense surface.
        {"name": "nearest_samples", "op": "nearest", "edges": 7.0, "n": 400001, "targets": 100003},
        # One working mesh of about 66 000 faces, labelled.
        {"name": "preprocess_fragment", "op": "preprocess", "edges": 7.0},
        # One join refined on meshes of about 800 000 faces.
        {"name": "refine_join", "op": "refine", "edges": 24.0},
        # 64 group poses of a 6-fragment pot.
        {"name": "group_adjoint", "op": "adjoint", "edges": 5.0, "cells": 6, "t": 12.0,
         "poses": 64},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["verify", "stage2", "stage2", "stage2", "resident", "icp", "stage1", "inside",
                     "distance", "nearest", "preprocess", "refine", "adjoint"])
    edges = round(rng.uniform(4.0, 12.0), 3)
    if op in ("verify", "stage1"):
        return {"op": op, "edges": min(edges, 8.0) if op == "stage1" else edges}
    if op == "stage2" and rng.random() < 0.6:
        return {"op": op, "edges": edges, "cells": 0, "starts": int(_log(rng, 1, 130)),
                "early": rng.choice([0.0, 0.0, 0.15])}
    if op in ("stage2", "resident"):
        return {"op": op, "edges": round(rng.uniform(4.0, 7.0), 3), "cells": rng.randint(3, 7),
                "walls": 1 if op == "stage2" else rng.randint(1, 2),
                "starts": int(_log(rng, 4, 100)), "t": round(rng.uniform(10.0, 14.0), 3),
                "frac_per_t2": round(_log(rng, 60.0, 900.0), 2),
                "frac_max": int(_log(rng, 6000, 60000)), "early": rng.choice([0.0, 0.0, 0.15])}
    if op == "icp":
        return {"op": op, "edges": edges, "starts": int(_log(rng, 1, 130)),
                "k": rng.choice([0.04, 0.08, 0.2])}
    if op in ("inside", "distance"):
        return {"op": op, "edges": edges, "n": int(_log(rng, 100, 400000))}
    if op == "nearest":
        return {"op": op, "edges": edges, "n": int(_log(rng, 50, 800000)),
                "targets": int(_log(rng, 50, 300000))}
    if op == "preprocess":
        return {"op": op, "edges": edges}
    if op == "refine":
        return {"op": op, "edges": round(rng.uniform(8.0, 24.0), 3)}
    return {"op": op, "edges": round(rng.uniform(4.0, 6.0), 3), "cells": rng.randint(3, 6),
            "t": round(rng.uniform(10.0, 14.0), 3), "poses": int(_log(rng, 1, 100))}


# ---- inputs ---------------------------------------------------------------------------------

# Operations whose output sizes follow from the geometry itself: their fragments come from one
# generator seed and the case's seed places them (and draws poses and probes).
FIXED = {"stage1": 3, "refine": 3, "adjoint": 3}


def _fragments(case, seed):
    """The generated workload of a case: the cut slab, or the pots of a collection."""
    seed = FIXED.get(case["op"], seed)
    if not case.get("cells"):
        # (half of a pair's starts lie near the join: a rung takes that half)
        starts = case.get("starts", 4) * (2 if case["op"] == "icp" else 1)
        return synth.slab_collection(seed, edges_per_t=case["edges"], n_starts=starts)
    t, walls = case["t"], case.get("walls", 1)
    dens = case.get("frac_per_t2", 150.0)
    return synth.pot_collection(
        seed, walls=(t, 1.4 * t)[:walls], cells_per_wall=(case["cells"],) * walls,
        edges_per_t=(case["edges"] - 1.0, case["edges"] + 1.0), n_starts=case.get("starts", 4),
        frac_per_t2=(dens, 60.0)[:walls], frac_range=(1000, case.get("frac_max", 12000)))


def _samples(wl, case, seed):
    """n samples of B's faces laid near their true place on A (0.5 deg, 0.1 t off), with the pose
    that lays them: points f64 (n, 3) in B's frame, pose 4x4."""
    rng = np.random.default_rng(seed + 1)
    a, b = wl.fragments
    v = b.v.astype(np.float64)
    f = b.f.astype(np.int64)
    _, areas, _ = synth.face_geometry(v, f)
    faces = np.flatnonzero(b.frac) if case["op"] == "distance" else np.arange(len(f))
    pts, _ = synth.sample_on_faces(rng, v, f, areas, faces, case["n"])
    c = pts.mean(0)
    rot = synth.random_rotation(rng, 0.5)
    step = rng.normal(size=3)
    step *= 0.1 * b.t / np.linalg.norm(step)
    return np.ascontiguousarray(pts), wl.pairs[0].truth @ synth.rigid(rot, c - rot @ c + step)


def _placements(seed):
    """Two rigid poses a pair's fragments are moved by."""
    rng = np.random.default_rng(seed + 3)
    return [synth.rigid(synth.random_rotation(rng), rng.uniform(-100.0, 100.0, size=3))
            for _ in range(2)]


def _params(case):
    p = sherd.default_params()
    p.early_reject_tight = case.get("early", 0.0)
    return p


def prepare(case, seed):
    op = case["op"]
    ctx = context()
    wl = _fragments(case, seed)
    state = {"op": op, "ctx": ctx}
    if op in ("verify", "stage2", "resident", "icp", "adjoint"):
        dev = workload.to_device(ctx, wl)
        state["dev"] = dev
    if op == "verify":
        state["pose"] = wl.starts[0][0]
    elif op == "stage2":
        state["params"] = _params(case)
        state["out"] = np.zeros(dev.n_items, sherd.CANDIDATE)
    elif op == "resident":
        state["batch"] = ctx.batch(dev.pairs, dev.items, _params(case))
    elif op == "icp":
        state["source"] = wl.fragments[1].reg_p
        state["inits"] = wl.starts[0][:case["starts"]]
        s = dev.scales[0]
        state["distance"] = case["k"] * s.t * s.icp
    elif op == "stage1":
        frames = []
        for fr, m in zip(wl.fragments, _placements(seed)):
            k = preprocess.breaklines(ctx, fr.v.astype(np.float64), fr.f, fr.frac, fr.t).frames()
            r = m[:3, :3]
            frames.append(stage1.Frames(p=k.p @ r.T + m[:3, 3], ns=k.ns @ r.T, f=k.f @ r.T,
                                        dih=k.dih, sub=k.sub))
        sc = workload.pair_scales(wl)[0]
        state["pair"] = stage1.PairStage1(ctx, frames[0], frames[1], sc)
        state["seed"] = seed
    elif op in ("inside", "distance"):
        state["points"], state["pose"] = _samples(wl, case, seed)
        mesh = ctx.mesh(wl.fragments[0].v, wl.fragments[0].f)
        state["mesh"] = mesh if op == "inside" else mesh.subset(wl.fragments[0].frac)
        state["bound"] = 0.5 * wl.fragments[0].t
    elif op == "nearest":
        a = wl.fragments[0]
        rng = np.random.default_rng(seed + 2)
        v, f = a.v.astype(np.float64), a.f.astype(np.int64)
        areas = synth.face_geometry(v, f)[1]
        target, _ = synth.sample_on_faces(rng, v, f, areas, np.arange(len(f)), case["targets"])
        pts, pose = _samples(wl, case, seed)
        state["queries"] = pts @ pose[:3, :3].T + pose[:3, 3]
        state["target"] = target
        state["cloud"] = ctx.cloud(target)
        state["bound"] = 0.5 * a.t
    elif op == "preprocess":
        fr = wl.fragments[0]
        state.update(v=fr.v.astype(np.float64), v32=fr.v, f=fr.f, res=fr.res, t=fr.t, frac=fr.frac)
    elif op == "refine":
        state["meshes"] = []
        placed = _placements(seed)
        for fr, m in zip(wl.fragments, placed):
            state["meshes"].append((np.float32(fr.v @ m[:3, :3].T + m[:3, 3]).astype(np.float64),
                                    fr.f))
        state["centroids"] = [synth.face_geometry(v, f.astype(np.int64))[2]
                              for v, f in state["meshes"]]
        state["fragments"] = [(fr.frac, fr.t, fr.res) for fr in wl.fragments]
        world = workload.perturbed_group_poses(wl, 1, seed=seed + 1, rot_deg=0.1, trans_t=0.02)[1]
        state["poses"] = [w @ np.linalg.inv(m) for w, m in zip(world[0], placed)]
    elif op == "adjoint":
        group = workload.assembled_group(dev, wl)
        world = workload.perturbed_group_poses(wl, case["poses"], seed=seed + 1)[1]
        state["group"] = group
        state["poses"], state["inverses"] = group.relative(world)
    state["wl"] = wl
    return state


# ---- one pass -------------------------------------------------------------------------------

SCORES = [n for n, _ in sherd.Scores._fields_]


def _candidates(c):
    r, s = c["rungs"], c["scores"]
    return {"transform": r["transform"], "fitness": r["fitness"], "rmse": r["inlier_rmse"],
            "correspondences": r["correspondences"], "iterations": r["iterations"],
            "converged": r["converged"], "accepted": c["accepted"], "status": c["status"],
            **{"score_" + k: s[k] for k in SCORES}}


def _registrations(r):
    return {"transform": r["transform"], "fitness": r["fitness"], "rmse": r["inlier_rmse"],
            "correspondences": r["correspondences"], "iterations": r["iterations"],
            "converged": r["converged"]}


def run(state):
    op, ctx = state["op"], state["ctx"]
    if op == "verify":
        dev = state["dev"]
        s = ctx.verify(dev.surfaces[0], dev.surfaces[1], state["pose"], dev.scales[0])
        return {k: getattr(s, k) for k in SCORES}
    if op == "stage2":
        dev = state["dev"]
        return _candidates(ctx.ladder_verify_batch(dev.pairs, dev.items, state["params"],
                                                   out=state["out"]))
    if op == "resident":
        state["batch"].run()
        return _candidates(sherd.candidates(state["batch"].results()))
    if op == "icp":
        return _registrations(ctx.icp_rung_array(state["source"], state["dev"].reg_targets[0],
                                                 state["inits"], state["distance"]))
    if op == "stage1":
        r = state["pair"].run(seed=state["seed"])
        return {"pa": r.hypotheses.pa, "pb": r.hypotheses.pb, "poses": r.hypotheses.poses,
                "coarse": r.coarse, "kept": r.kept, "transforms": r.transforms,
                "scores": r.scores, "kept2": r.kept2}
    if op == "inside":
        depth, inside = ctx.inside(state["mesh"], state["points"], state["pose"])
        return {"depth": depth, "inside": inside}
    if op == "distance":
        return {"distance": ctx.bounded_distance(state["mesh"], state["points"], state["pose"],
                                                 state["bound"])}
    if op == "nearest":
        idx, dist = state["cloud"].nearest_below(state["queries"], state["bound"])
        return {"idx": idx, "dist": dist}
    if op == "preprocess":
        mesh = ctx.mesh(state["v32"], state["f"])
        normals, areas, centroids = ctx.face_geometry(state["v"], state["f"])
        (thick, mode), t_hit, prim = ctx.thickness(mesh, centroids, normals, return_hits=True)
        labels, _ = ctx.segment(mesh, state["v"], state["f"], thick, state["res"])
        brk = ctx.breaklines(state["v"], state["f"], state["frac"], state["t"])
        return {"normals": normals, "areas": areas, "centroids": centroids, "thick": thick,
                "mode": mode, "t_hit": t_hit, "prim": prim, "labels": labels,
                "brk_p": brk["p"], "brk_ns": brk["ns"], "brk_nf": brk["nf"], "brk_f": brk["f"],
                "brk_dih": brk["dih"], "brk_valid": brk["valid"]}
    if op == "refine":
        pieces = [refine.RefinePiece(t, res, refine.fracture_cloud(ctx, v, f, c, frac, t, res))
                  for (v, f), c, (frac, t, res) in zip(state["meshes"], state["centroids"],
                                                       state["fragments"])]
        out = refine.refine_joins(ctx, pieces, state["poses"], [[0, 1]], [(0, 1)])
        join = out.joins[0]
        return {"idx": [p.cloud.idx for p in pieces], "points": [p.cloud.points for p in pieces],
                "normals": [p.cloud.normals for p in pieces], "pose": out.poses[1],
                "rungs": join.rungs, "fitness": join.fitness, "rmse": join.rmse_t}
    group = state["group"]
    values, grads = ctx.adjoint(group.edges, state["poses"], state["inverses"], group.opts)
    return {"values": values, "grads": grads}


# ---- the least work -------------------------------------------------------------------------

def work(case):
    """Inputs read once, outputs written once, and the arithmetic of every point's transform,
    distance and accumulation (one pass per rung, the fewest an ICP rung makes is two)."""
    wl = _fragments(case, 1)
    op, fr = case["op"], wl.fragments
    mesh = sum(len(x.v) * 12 + len(x.f) * 12 for x in fr)
    if op in ("verify", "stage2", "resident", "icp"):
        samples = sum(24 * (len(x.pf) + len(x.s) + 2 * len(x.brk_p) + 2 * len(x.margin_p)) +
                      48 * (len(x.reg_p) + len(x.pf)) for x in fr)
        if op == "verify":
            points = sum(len(x.pf) + len(x.s) + len(x.brk_p) + len(x.margin_p) for x in fr)
            return {"bytes": mesh + samples, "flops": 40 * points}
        if op == "icp":
            n = len(fr[1].reg_p)
            return {"bytes": 48 * (n + len(fr[0].reg_p)) + 300 * case["starts"],
                    "flops": 2 * 150 * n * case["starts"]}
        flops = 0
        for p, s in zip(wl.pairs, wl.starts):
            a, b = fr[p.a], fr[p.b]
            icp = 2 * 2 * 150 * (len(b.reg_p) + len(b.pf))
            ver = 40 * (len(a.pf) + len(b.pf) + len(a.s) + len(b.s) + len(a.brk_p) +
                        len(b.margin_p))
            flops += len(s) * (icp + ver)
        return {"bytes": mesh + samples + 944 * wl.n_items, "flops": flops}
    if op == "stage1":
        n = 2 * sum(len(x.brk_p) for x in fr)
        return {"bytes": 80 * n + 144 * n * n // 16, "flops": 60 * 40 * n * n // 16}
    if op in ("inside", "distance"):
        return {"bytes": mesh // 2 + 32 * case["n"], "flops": 60 * case["n"]}
    if op == "nearest":
        return {"bytes": 36 * case["n"] + 24 * case["targets"], "flops": 8 * case["n"]}
    if op == "preprocess":
        nf, nv = len(fr[0].f), len(fr[0].v)
        return {"bytes": 24 * nv + 12 * nf + (56 + 8 + 1) * nf, "flops": 500 * nf}
    if op == "refine":
        nv, nf = sum(len(x.v) for x in fr), sum(len(x.f) for x in fr)
        return {"bytes": 24 * nv + (12 + 24 + 1) * nf, "flops": 60 * nf}
    edges = sum(p.adjacent for p in wl.pairs)
    points = sum(2 * len(fr[p.b].pf) + len(fr[p.a].pf) for p in wl.pairs if p.adjacent)
    return {"bytes": mesh + sum(72 * len(x.pf) for x in fr) + case["poses"] * edges * 536,
            "flops": 120 * points * case["poses"]}


# ---- the answers in 64 bits -------------------------------------------------------------------

def _gpu(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device="cuda")


def _nearest(q, p, rows=None):
    """Brute force: each query's nearest point (the lowest index on a tie) and squared distance."""
    rows = rows or max(1, (1 << 27) // max(len(p), 1))
    idx, best = [], []
    for c in q.split(rows):
        d = (c[:, None, 0] - p[None, :, 0]).square_()
        for k in (1, 2):
            d += (c[:, None, k] - p[None, :, k]).square_()
        m, i = d.min(1)
        idx.append(i)
        best.append(m)
    return torch.cat(idx), torch.cat(best)


def _closest(p, a, b, c):
    """The closest points of triangles abc to points p (broadcast, last axis 3)."""
    ab, ac, ap = b - a, c - a, p - a
    dot = lambda u, v: (u * v).sum(-1)
    d1, d2 = dot(ab, ap), dot(ac, ap)
    bp, cp = p - b, p - c
    d3, d4, d5, d6 = dot(ab, bp), dot(ac, bp), dot(ab, cp), dot(ac, cp)
    va, vb, vc = d3 * d6 - d5 * d4, d5 * d2 - d1 * d6, d1 * d4 - d3 * d2
    den = va + vb + vc
    v, w = vb / den, vc / den
    zero = torch.zeros_like(v)
    for at, sv, sw in (
            ((va <= 0) & (d4 - d3 >= 0) & (d5 - d6 >= 0),
             1 - (d4 - d3) / (d4 - d3 + d5 - d6), (d4 - d3) / (d4 - d3 + d5 - d6)),
            ((vb <= 0) & (d2 >= 0) & (d6 <= 0), zero, d2 / (d2 - d6)),
            ((d6 >= 0) & (d5 <= d6), zero, zero + 1),
            ((vc <= 0) & (d1 >= 0) & (d3 <= 0), d1 / (d1 - d3), zero),
            ((d3 >= 0) & (d4 <= d3), zero + 1, zero),
            ((d1 <= 0) & (d2 <= 0), zero, zero)):
        v, w = torch.where(at, sv, v), torch.where(at, sw, w)
    return a + ab * v[..., None] + ac * w[..., None]


def _mesh_nearest(p, tri, rows=None):
    """Brute force: each point's distance to the nearest triangle, and the closest point on it."""
    rows = rows or max(1, (1 << 22) // max(len(tri), 1))
    dist, at = [], []
    for c in p.split(rows):
        q = _closest(c[:, None], tri[None, :, 0], tri[None, :, 1], tri[None, :, 2])
        d = (q - c[:, None]).square().sum(-1)
        m, i = d.min(1)
        dist.append(m.sqrt())
        at.append(q[torch.arange(len(c), device=q.device), i])
    return torch.cat(dist), torch.cat(at)


def _parity(p, tri, axis):
    """Whether the +axis ray from each point crosses the triangles an odd number of times."""
    u, v = (axis + 1) % 3, (axis + 2) % 3
    odd = []
    for c in p.split(max(1, (1 << 25) // len(tri))):
        cu, cv, cw = (c[:, None, k] for k in (u, v, axis))
        s = []
        for k in range(3):
            a, b = tri[:, k], tri[:, (k + 1) % 3]
            s.append((b[:, u] - a[:, u]) * (cv - a[:, v]) - (b[:, v] - a[:, v]) * (cu - a[:, u]))
        area = s[0] + s[1] + s[2]
        hit = ((s[0] >= 0) & (s[1] >= 0) & (s[2] >= 0)) | ((s[0] <= 0) & (s[1] <= 0) & (s[2] <= 0))
        depth = (s[1] * tri[:, 0, axis] + s[2] * tri[:, 1, axis] + s[0] * tri[:, 2, axis]) / area
        odd.append((hit & (area != 0) & (depth > cw)).sum(1) % 2)
    return torch.cat(odd)


def _icp(source, target, normals, init, distance, iterations):
    """registration_icp, point-to-plane, one start: (transform, fitness, rmse)."""
    t = _gpu(init).reshape(4, 4)
    fit = rmse = 0.0
    for it in range(iterations + 1):
        x = source @ t[:3, :3].T + t[:3, 3]
        j, d2 = _nearest(x, target)
        m = d2 < distance * distance
        x, q, n = x[m], target[j[m]], normals[j[m]]
        count = int(m.sum())
        f, r = count / len(source), math.sqrt(float(d2[m].sum()) / count) if count else 0.0
        done = it > 0 and abs(f - fit) < 1e-6 and abs(r - rmse) < 1e-6
        fit, rmse = f, r
        if done or it == iterations or not count:
            break
        row = torch.cat([torch.linalg.cross(x, n), n], 1)
        res = ((x - q) * n).sum(1)
        s = torch.linalg.solve(row.T @ row, -(row.T @ res)).cpu().numpy()
        (sa, ca), (sb, cb), (sg, cg) = ((math.sin(k), math.cos(k)) for k in s[:3])
        rot = (np.array([[cg, -sg, 0], [sg, cg, 0], [0, 0, 1]]) @
               np.array([[cb, 0, sb], [0, 1, 0], [-sb, 0, cb]]) @
               np.array([[1, 0, 0], [0, ca, -sa], [0, sa, ca]]))
        u = np.eye(4)
        u[:3, :3], u[:3, 3] = rot, s[3:]
        t = _gpu(u) @ t
    return t.cpu().numpy().reshape(16), fit, rmse


def _triangles(v, f):
    return _gpu(np.asarray(v, np.float32).astype(np.float64)[f.astype(np.int64)])


def _moved(points, pose):
    pose = _gpu(pose)
    return _gpu(points) @ pose[:3, :3].T + pose[:3, 3]


def exact(case, seed):
    op = case["op"]
    wl = _fragments(case, seed)
    fr = wl.fragments
    if op == "verify":
        a, b = fr
        sc = workload.pair_scales(wl)[0]
        pose = wl.starts[0][0]
        out = {k: None for k in SCORES}
        tris = [_triangles(x.v, x.f[x.frac.astype(bool)]) for x in fr]
        sides = {"a": (a.pf, np.linalg.inv(pose), tris[1], a.frac_area),
                 "b": (b.pf, pose, tris[0], b.frac_area)}
        for k, (p, m, tri, area) in sides.items():
            d = _mesh_nearest(_moved(p, m), tri)[0]
            near = d[d < sc.facing]
            if len(near) >= 20:
                out["gap_" + k] = float(np.median(near.cpu().numpy())) / sc.t
                out["contact_" + k] = float((d < 2 * sc.tight).double().mean()) * area / sc.t ** 2
        return out
    if op == "icp":
        a, b = fr
        s = workload.pair_scales(wl)[0]
        src, tgt, nrm = _gpu(b.reg_p), _gpu(a.reg_p), _gpu(a.reg_n)
        regs = [_icp(src, tgt, nrm, t, case["k"] * s.t * s.icp, 30) for t in wl.starts[0][:case["starts"]]]
        return {"transform": np.stack([r[0] for r in regs]),
                "fitness": np.array([r[1] for r in regs]), "rmse": np.array([r[2] for r in regs])}
    if op == "inside":
        pts, pose = _samples(wl, case, seed)
        if case["n"] * len(fr[0].f) > 6e9:
            return None
        p, tri = _moved(pts, pose).float().double(), _triangles(fr[0].v, fr[0].f)
        votes = _parity(p, tri, 0) + _parity(p, tri, 1) + _parity(p, tri, 2)
        depth = torch.zeros(len(p), dtype=torch.float64, device="cuda")
        hit = votes >= 2
        depth[hit] = _mesh_nearest(p[hit], tri)[0]
        return {"depth": depth.cpu().numpy(), "inside": None}
    if op == "distance":
        tri = _triangles(fr[0].v, fr[0].f[fr[0].frac.astype(bool)])
        if case["n"] * len(tri) > 3e9:
            return None
        pts, pose = _samples(wl, case, seed)
        d = _mesh_nearest(_moved(pts, pose), tri)[0]
        return {"distance": torch.where(d <= 0.5 * fr[0].t, d, torch.inf).cpu().numpy()}
    if op == "nearest":
        if case["n"] * case["targets"] > 5e10:
            return None
        a = fr[0]
        rng = np.random.default_rng(seed + 2)
        v, f = a.v.astype(np.float64), a.f.astype(np.int64)
        areas = synth.face_geometry(v, f)[1]
        target, _ = synth.sample_on_faces(rng, v, f, areas, np.arange(len(f)), case["targets"])
        pts, pose = _samples(wl, case, seed)
        i, d2 = _nearest(_gpu(pts @ pose[:3, :3].T + pose[:3, 3]), _gpu(target))
        d = d2.sqrt()
        return {"idx": None, "dist": torch.where(d < 0.5 * a.t, d, torch.inf).cpu().numpy()}
    if op == "preprocess":
        v, f = fr[0].v.astype(np.float64), fr[0].f.astype(np.int64)
        n = np.cross(v[f[:, 1]] - v[f[:, 0]], v[f[:, 2]] - v[f[:, 0]])
        length = np.linalg.norm(n, axis=1)
        return {"normals": n / np.maximum(length, 1e-12)[:, None], "areas": 0.5 * length,
                "centroids": v[f].mean(1)}
    if op == "adjoint":
        return _exact_adjoint(wl, case, seed)
    return None  # chains of rungs, whose answers a last bit of one pass can turn


def _exact_adjoint(wl, case, seed):
    fr = wl.fragments
    edges = [(k, p.a, p.b) for k, p in enumerate(wl.pairs) if p.adjacent]
    tris = {i: _triangles(fr[i].v, fr[i].f[fr[i].frac.astype(bool)]) for _, a, b in edges
            for i in (a, b)}
    pairs = sum(len(fr[b].pf) * len(tris[a]) + len(fr[a].pf) * len(tris[b]) for _, a, b in edges)
    if case["poses"] * pairs > 2e10:
        return None
    scales = workload.pair_scales(wl)
    world = workload.perturbed_group_poses(wl, case["poses"], seed=seed + 1)[1]
    inv = np.linalg.inv(world)
    values = np.zeros((case["poses"], len(edges), 5))
    grads = np.zeros((case["poses"], len(edges), 5, 6))

    def twist(p, g):
        return torch.cat([torch.linalg.cross(p, g), g], 1).sum(0).cpu().numpy()

    for e, (k, a, b) in enumerate(edges):
        sc = scales[k]
        w, r = 0.01 * sc.t, 0.2 * sc.t * sc.icp
        window = sc.facing + 30.0 * w
        tgt, nrm = _gpu(fr[a].pf), _gpu(fr[a].pf_n)
        for g in range(case["poses"]):
            t, ti = inv[g, a] @ world[g, b], inv[g, b] @ world[g, a]
            x = _moved(fr[b].pf, t)
            j, d2 = _nearest(x, tgt)
            m = d2 < r * r
            x, q, n = x[m], tgt[j[m]], nrm[j[m]]
            res = ((x - q) * n).sum(1, keepdim=True)
            values[g, e, 0] = 0.5 * float(res.square().sum())
            grads[g, e, 0] = twist(x, res * n)
            for o, pts, pose, tri in ((1, fr[b].pf, t, tris[a]), (3, fr[a].pf, ti, tris[b])):
                x = _moved(pts, pose)
                d, q = _mesh_nearest(x, tri)
                m = d <= window
                x, dv = x[m], x[m] - q[m]
                d = (dv.square().sum(1, keepdim=True) + 0.01 * w * w).sqrt()
                for z, limit in ((0, sc.tight), (1, sc.facing)):
                    s = torch.sigmoid((limit - d) / w)
                    values[g, e, o + z] = float(s.sum())
                    grads[g, e, o + z] = twist(x, -s * (1 - s) / (w * d) * dv)
    return {"values": values, "grads": grads}
