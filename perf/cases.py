"""Performance cases: the work a program asks of the framework, over its sizes.

A case is a dict of plain values. Its `kind` names the public entry points:

  frame        NonRigidSolver.set_solver_input / solve_non_rigid_alignment /
               solved_node_se3: one frame of a live reconstruction
  batch        StreamedBatch.set_input / solve / node_se3_async: many
               independent solves as replayed graphs
  warp         SurfelNodeDeformer forward and inverse warps of the surfels
  node_error   NonRigidSolver.compute_alignment_error_on_nodes with its maps
  solver_maps  SolverMapRenderer.draw_solver_maps_with_recent_observation
  spmv         mvdr_bsr6_spmv_dot_noalloc on a matrix the caller owns

The inputs are synthetic scenes of the shapes the benchmark uses (a sphere, a
torso, an articulated body; the same camera rings, depth noise, warp-field
perturbation and skinning rule), ray-cast on the GPU from the seed. `exact`
restates each case in float64 with torch.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from multiviewdynrecon_b200 import abi, check, lib, synth
from multiviewdynrecon_b200.deform import SurfelNodeDeformer
from multiviewdynrecon_b200.solver import DeviceScene, NonRigidSolver, StreamedBatch
from multiviewdynrecon_b200.solver_maps import SolverMapRenderer

DEV = "cuda"
F64 = torch.float64
EMPTY = 0xFFFFFFFF  # an index-map pixel without a surfel


# ------------------------------------------------------------------ cases ----

def _frame(name, shape, views, width, height, nodes, gn, pcg, **more):
    case = dict(name=name, kind="frame", shape=shape, views=views, width=width, height=height, nodes=nodes, gn=gn,
                pcg=pcg, precision="mixed", mode="materialized", focal=1.0, features=0, cross=0, foreground=False,
                density=False, pairs=False, global_iterations=1 << 20)
    case.update(more)
    return case


def listed():
    return [
        # the smallest frame: one low-resolution camera, a coarse node graph;
        # launches and latency decide
        _frame("frame_small", "sphere", 1, 320, 240, 500, 3, 10),
        # the plain single-view method in plain FP32
        _frame("frame_sphere_fp32", "sphere", 1, 640, 480, 2048, 3, 10, precision="fp32"),
        # the ordinary live frame: three cameras, every term
        _frame("frame_torso", "torso", 3, 640, 480, 4096, 5, 15, features=1000, cross=2000, foreground=True),
        # odd sizes with the colour term: device-selected feature pairs, the
        # global then the local penalty phase
        _frame("frame_density_odd", "torso", 2, 633, 475, 3001, 4, 12, features=777, cross=1333, foreground=True,
               density=True, pairs=True, global_iterations=2),
        # the matrix-free operator
        _frame("frame_matrix_free", "torso", 3, 640, 480, 4096, 5, 15, features=1000, cross=2000, foreground=True,
               mode="matrix_free"),
        # the largest frame: an articulated body filling five HD cameras,
        # about 4M dense terms
        _frame("frame_body", "body", 5, 1280, 720, 32768, 8, 20, cross=4000, focal=5.0),
        # offline batches: sixteen initial fields of one subject, and subjects
        # of uneven sizes
        dict(_frame("batch_torso", "torso", 3, 640, 480, 4096, 5, 15, features=1000, cross=2000, foreground=True),
             kind="batch", count=16, min_nodes=4096),
        dict(_frame("batch_uneven", "torso", 4, 640, 480, 15680, 5, 15, features=1000, cross=2000, foreground=True),
             kind="batch", count=8, min_nodes=1281),
        # after the solve: all surfels of the body moved to the live frame and back
        dict(name="warp_body", kind="warp", surfels=4000000, nodes=32768),
        # node alignment errors and both error maps of five HD views
        dict(_frame("node_error_body", "body", 5, 1280, 720, 32768, 0, 0, focal=5.0), kind="node_error"),
        # the renderer's solver maps of the body's surfels, sized points in view 0
        dict(_frame("solver_maps_body", "body", 5, 1280, 720, 32768, 0, 0, focal=5.0), kind="solver_maps",
             sized=True),
        # the operator step on a caller's block-sparse matrix (ragged rows)
        dict(name="spmv_odd", kind="spmv", rows=4099, per_row=19),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["batch"] * 2 + ["warp", "node_error", "solver_maps", "spmv"])
    if kind == "warp":
        return dict(kind="warp", surfels=_log_int(rng, 20000, 4000000), nodes=_log_int(rng, 500, 32768))
    if kind == "spmv":
        return dict(kind="spmv", rows=_log_int(rng, 500, 40000), per_row=rng.randint(8, 24))
    width = _log_int(rng, 320, 1280)
    height = int(width * rng.choice([0.5625, 0.75])) + rng.randint(-3, 3)
    case = _frame("", rng.choice(["sphere", "torso", "torso", "body"]), rng.randint(1, 5), width, height, 0, 0, 0)
    del case["name"]
    case["focal"] = 5.0 if case["shape"] == "body" else 1.0
    if kind == "batch":
        case.update(kind="batch", shape="torso", focal=1.0, count=rng.randint(3, 12), views=rng.randint(1, 4),
                    width=_log_int(rng, 320, 640))
        case["height"] = int(case["width"] * 0.75)
    # a node carries a few hundred terms (each pixel counts for four nodes)
    terms = 4.0 * case["views"] * case["width"] * case["height"] * _coverage(case)
    lo = max(500, int(terms / 500))
    case["nodes"] = min(32768, _log_int(rng, lo, max(lo + 1, min(32768, int(terms / 60)))))
    if kind in ("node_error", "solver_maps"):
        case["kind"] = kind
        if kind == "solver_maps":
            case["sized"] = rng.random() < 0.5
        return case
    case.update(gn=rng.randint(3, 6), pcg=rng.randint(10, 18), foreground=rng.random() < 0.6,
                features=rng.choice([0, rng.randint(200, 1200)]),
                cross=rng.randint(300, 2500) if case["views"] > 1 else 0)
    if kind == "batch":
        case["nodes"] = min(case["nodes"], 12000)
        case["min_nodes"] = max(300, case["nodes"] // rng.randint(1, 2))
        return case
    case["precision"] = rng.choice(["mixed", "mixed", "mixed", "fp32"])
    if rng.random() < 0.2 and terms < 3e6:
        case["mode"] = "matrix_free"
    if rng.random() < 0.3:
        case.update(density=True, global_iterations=2)
    case["pairs"] = case["features"] > 0 and rng.random() < 0.3
    return case


# ----------------------------------------------------------------- scenes ----

def _shapes(shape, rng):
    """Ellipsoids (centre, semi-axes, rotation), jittered by the seed."""
    eye = np.eye(3)

    def axes(*a):
        return np.array(a) * (1.0 + rng.uniform(-0.04, 0.04, 3))

    if shape == "sphere":
        return [(np.array([0.0, 0.0, 2.5]), axes(1.0, 1.0, 1.0), eye)], 2.5
    if shape == "torso":
        return [(np.array([0.0, 0.0, 1.3]), axes(0.25, 0.6, 0.15), eye)], 1.3
    centre = np.array([0.0, 0.0, 2.2])
    parts = [(centre, axes(0.25, 0.45, 0.15), eye)]
    for anchor, d in (((-0.3, -0.3), (-1, 0.2)), ((0.3, -0.3), (1, 0.2)), ((-0.12, 0.45), (-0.15, 1)),
                      ((0.12, 0.45), (0.15, 1))):
        d = np.array([d[0], d[1], 0.0]) / math.hypot(*d)
        R = synth.rodrigues(np.array([0, 0, 1.0]) * math.radians(rng.uniform(-30, 30)))
        d = R @ d
        side = np.array([-d[1], d[0], 0.0])
        parts.append((centre + np.array([*anchor, 0.0]) + 0.27 * d, axes(0.06, 0.33, 0.06),
                      np.stack([side, d, np.cross(side, d)], 1)))
    return parts, 2.2


def _cameras(views, distance):
    """Camera-to-frame-0 poses on a ring around the subject; view 0 is frame 0."""
    centre = np.array([0.0, 0.0, distance])
    cams = [(np.eye(3), np.zeros(3))]
    for k in range(1, views):
        a = 2 * math.pi * k / views
        cams.append(synth.look_at(centre + distance * np.array([math.sin(a), 0.0, -math.cos(a)]), centre))
    return cams


def _cast(parts, R, o, W, H, f, device):
    """Nearest hit of every pixel's ray: (valid, point, normal), frame 0."""
    u = torch.arange(W, dtype=F64, device=device)
    v = torch.arange(H, dtype=F64, device=device)
    d = torch.stack(torch.broadcast_tensors(((u - W / 2) / f)[None], ((v - H / 2) / f)[:, None],
                                            torch.ones((), dtype=F64, device=device)), -1).reshape(-1, 3)
    d = d @ torch.as_tensor(R, dtype=F64, device=device).T
    o = torch.as_tensor(o, dtype=F64, device=device)
    best = torch.full((len(d),), math.inf, dtype=F64, device=device)
    normal = torch.zeros_like(d)
    for c, ax, Rp in parts:
        M = torch.as_tensor(Rp / ax[None], dtype=F64, device=device)  # to the unit sphere
        c = torch.as_tensor(c, dtype=F64, device=device)
        dl, ol = d @ M, (o - c) @ M
        A, B, Q = (dl * dl).sum(1), dl @ ol, ol @ ol - 1.0
        disc = B * B - A * Q
        t = (-B - disc.clamp(min=0).sqrt()) / A
        hit = (disc > 0) & (t > 0) & (t < best)
        n = (ol + t[:, None] * dl) @ M.T
        n = n / n.norm(dim=1, keepdim=True)
        best = torch.where(hit, t, best)
        normal = torch.where(hit[:, None], n, normal)
    valid = best.isfinite()
    return valid, o + torch.where(valid, best, 0.0)[:, None] * d, normal


_COVERAGE = {}


def _coverage(case):
    """Share of the pixels that see the subject (nominal shape, view 0)."""
    key = (case["shape"], case["focal"])
    if key not in _COVERAGE:
        parts, dist = _shapes(case["shape"], np.random.default_rng(0))
        valid, _, _ = _cast(parts, np.eye(3), np.zeros(3), 96, 72, 570.0 * 96 / 640 * case["focal"], "cpu")
        _COVERAGE[key] = float(valid.double().mean())
    return _COVERAGE[key]


def _thin(points, count, gen):
    """`count` points at about equal spacing: one per voxel, in random order."""
    pts = points[torch.randperm(len(points), generator=gen, device=DEV)[: 128 * count]]
    lo, hi = 1e-4, 1.0
    for _ in range(14):
        s = math.sqrt(lo * hi)
        key = torch.floor((pts + 10.0) / s).to(torch.int64)
        key = (key[:, 0] * 2000003 + key[:, 1]) * 2000003 + key[:, 2]
        _, inv = torch.unique(key, return_inverse=True)
        n = int(inv.max()) + 1
        if n >= count:
            first = torch.full((n,), len(pts), dtype=torch.int64, device=DEV)
            first.scatter_reduce_(0, inv, torch.arange(len(pts), device=DEV), "amin")
            keep, lo = first, s
            if n <= 1.05 * count:
                break
        else:
            hi = s
    return pts[keep[torch.randperm(len(keep), generator=gen, device=DEV)[:count]]]


def _nearest(points, nodes, k):
    """The k nearest nodes of every point (squared distances, ids), by way of
    the 32 nodes nearest to the point's voxel."""
    spacing = float(torch.cdist(nodes[:512], nodes).topk(2, largest=False)[0][:, 1].mean())
    key = torch.floor((points + 10.0) / spacing).to(torch.int64)
    _, inv = torch.unique((key[:, 0] * 2000003 + key[:, 1]) * 2000003 + key[:, 2], return_inverse=True)
    cells = int(inv.max()) + 1
    centre = torch.zeros((cells, 3), dtype=F64, device=DEV).index_add_(0, inv, points)
    centre /= torch.bincount(inv, minlength=cells)[:, None]
    near = torch.cat([torch.cdist(c, nodes).topk(min(32, len(nodes)), largest=False)[1] for c in centre.split(2048)])
    d2, ids = [], []
    for p, c in zip(points.split(1 << 19), inv.split(1 << 19)):
        cand = near[c]
        d = ((nodes[cand] - p[:, None]) ** 2).sum(-1)
        v, j = d.topk(k, largest=False)
        d2.append(v)
        ids.append(cand.gather(1, j))
    return torch.cat(d2), torch.cat(ids)


def _skin(points, nodes, radius):
    d2, ids = _nearest(points, nodes, 4)
    w = torch.exp(-d2 / (2.0 * radius * radius))
    return ids, w / w.sum(1, keepdim=True).clamp(min=1e-30)


def _blur(m, sigma):
    r = int(4 * sigma + 0.5)
    x = torch.arange(-r, r + 1, dtype=F64, device=DEV)
    k = torch.exp(-x * x / (2 * sigma * sigma))
    k = (k / k.sum())[None, None]
    m = torch.nn.functional.pad(m[None, None], (r, r, r, r), mode="replicate")
    m = torch.nn.functional.conv2d(torch.nn.functional.conv2d(m, k[:, :, :, None]), k[:, :, None])
    return m[0, 0]


def _gradient(m):
    gy, gx = torch.gradient(m)
    return torch.stack([gx, gy], -1)


def _warp_field(nodes, gen):
    """The initial warp field: 2 degrees and 5 mm of noise about each node."""
    n = len(nodes)
    w = torch.randn((n, 3), generator=gen, device=DEV, dtype=F64) * math.radians(2.0)
    t = torch.randn((n, 3), generator=gen, device=DEV, dtype=F64) * 0.005
    w, t, p = w.cpu().numpy(), t.cpu().numpy(), nodes.cpu().numpy()
    R = synth.rodrigues_batch(w)
    return synth.se3_to_dq(R, p - np.einsum("nij,nj->ni", R, p) + t)


def _np32(t):
    return t.to(torch.float32).cpu().numpy()


def _scene(case, seed, nodes=None, views=None):
    """A synth.Scene of the case's shape: host arrays, as a capture pipeline
    hands them over."""
    nodes, views = nodes or case["nodes"], views or case["views"]
    W, H, radius = case["width"], case["height"], 0.025
    rng = np.random.default_rng(seed)
    gen = torch.Generator(DEV)
    gen.manual_seed(int(rng.integers(1 << 60)))
    parts, distance = _shapes(case["shape"], rng)
    cams = _cameras(views, distance)
    f = 570.0 * W / 640.0 * case["focal"]
    Rw, tw = synth.rodrigues(rng.normal(0, math.radians(0.3), 3)), rng.normal(0, 0.002, 3)  # rigid tracking
    Rwt, twt = torch.as_tensor(Rw, device=DEV), torch.as_tensor(tw, device=DEV)

    def noise(n, s):
        return torch.randn(n, generator=gen, device=DEV, dtype=F64) * s

    hits = [_cast(parts, R, o, W, H, f, DEV) for R, o in cams]
    vids = [h[0].nonzero()[:, 0] for h in hits]
    surfels = torch.cat([h[1][i] for h, i in zip(hits, vids)])
    normals = torch.cat([h[2][i] for h, i in zip(hits, vids)])
    node = _thin(surfels, nodes, gen)
    knn, w = _skin(surfels, node, radius)
    edges = torch.stack([torch.arange(nodes, device=DEV).repeat_interleave(8),
                         _nearest(node, node, 9)[1][:, 1:].reshape(-1)], 1)
    out, base, targets = [], 0, []
    for (R, o), (valid, p, n), vid in zip(cams, hits, vids):
        Rt, ot = torch.as_tensor(R, dtype=F64, device=DEV), torch.as_tensor(o, dtype=F64, device=DEV)

        def image(x, fill=0.0, dtype=F64):
            m = torch.full((H * W, x.shape[1]), fill, dtype=dtype, device=DEV)
            m[vid] = x.to(dtype)
            return m.reshape(H, W, -1)

        pv, nv = p[vid], n[vid]
        one = torch.ones((len(vid), 1), dtype=F64, device=DEV)
        live = (pv @ Rwt.T + twt - ot) @ Rt
        live = live * (1.0 + noise(len(vid), 0.002) / live[:, 2])[:, None]
        grey = 0.5 + 0.3 * torch.sin(9.0 * pv[:, :1] + 4.0 * pv[:, 1:2]) * torch.cos(7.0 * pv[:, 2:])
        index = torch.full((H * W,), EMPTY, dtype=torch.int64, device=DEV)
        index[vid] = base + torch.arange(len(vid), device=DEV)
        mask = _blur(1.0 - valid.reshape(H, W).to(F64), 2.0)
        dens = _blur(image(grey + noise((len(vid), 1), 0.005))[..., 0], 1.0)
        obs_v = image(torch.cat([live, one], 1))
        targets.append(obs_v.reshape(-1, 4)[:, :3])
        out.append(synth.View(
            reference_vertex_map=_np32(image(torch.cat([(pv - ot) @ Rt, one], 1))),
            reference_normal_map=_np32(image(torch.cat([nv @ Rt, one * radius * 0.1], 1))),
            index_map=index.cpu().numpy().astype(np.uint32).reshape(H, W),
            vertex_confidence_map=_np32(obs_v),
            normal_radius_map=_np32(image(torch.cat([nv @ Rwt.T @ Rt, one * 0.002], 1))),
            filtered_foreground_mask=_np32(mask), foreground_mask_gradient=_np32(_gradient(mask)),
            intrinsic=np.array([W / 2, H / 2, f, f], np.float32), world2camera=synth.mat34_pack(Rw, tw),
            initial_camera_se3=synth.mat34_pack(R, o),
            normalized_rgb_map=_np32(image(torch.cat([grey, grey, grey, one], 1))) if case["density"] else None,
            density_map=_np32(dens) if case["density"] else None,
            density_gradient_map=_np32(_gradient(dens)) if case["density"] else None))
        base += len(vid)

    def correspondences(src, tgt):
        one = torch.ones((len(src), 1), dtype=F64, device=DEV)
        return synth.Correspondences(_np32(torch.cat([tgt, one], 1)), _np32(torch.cat([surfels[src], one], 1)),
                                     knn[src].cpu().numpy().astype(np.uint16), _np32(w[src]))

    def frame0(pixels, v):
        """Observed points of view v's pixels in frame 0, rigid motion undone."""
        R, o = (torch.as_tensor(x, dtype=F64, device=DEV) for x in cams[v])
        return (targets[v][pixels] @ R.T + o - twt) @ Rwt

    starts = np.cumsum([0] + [len(i) for i in vids])
    src, tgt = [], []
    for v in range(views if case["features"] and not case["pairs"] else 0):  # 5 % outliers
        pick = torch.randperm(len(vids[v]), generator=gen, device=DEV)[: case["features"]]
        t = frame0(vids[v][pick], v)
        bad = torch.rand(len(pick), generator=gen, device=DEV) < 0.05
        src.append(starts[v] + pick)
        tgt.append(torch.where(bad[:, None], t + noise((len(pick), 3), 0.1), t))
    feature = correspondences(torch.cat(src), torch.cat(tgt)) if src else synth.Correspondences.empty()
    src, tgt = [], []
    for v in range(views if case["cross"] and views > 1 else 0):
        u = (v + 1) % views
        R, o = (torch.as_tensor(x, dtype=F64, device=DEV) for x in cams[u])
        pts = hits[v][1][vids[v]]
        pc = (pts - o) @ R
        x = torch.round(pc[:, 0] / pc[:, 2] * f + W / 2).to(torch.int64)
        y = torch.round(pc[:, 1] / pc[:, 2] * f + H / 2).to(torch.int64)
        ok = ((pc[:, 2] > 0.05) & (x >= 0) & (x < W) & (y >= 0) & (y < H)).nonzero()[:, 0]
        pix = y[ok] * W + x[ok]
        t = frame0(pix, u)
        close = ((t - pts[ok]).norm(dim=1) < 0.015) & (targets[u][pix][:, 2] > 0)
        ok, t = ok[close], t[close]
        pick = torch.randperm(len(ok), generator=gen, device=DEV)[: case["cross"]]
        src.append(starts[v] + ok[pick])
        tgt.append(t[pick])
    cross = correspondences(torch.cat(src), torch.cat(tgt)) if src else synth.Correspondences.empty()
    scene = synth.Scene(
        name=case["shape"], width=W, height=H, views=out, surfel_knn=knn.cpu().numpy().astype(np.uint16),
        surfel_knn_weight=_np32(w), node_se3=_warp_field(node, gen),
        canonical_nodes=_np32(torch.cat([node, torch.ones((nodes, 1), dtype=F64, device=DEV)], 1)),
        node_graph=edges.cpu().numpy().astype(np.uint16), feature=feature, cross_view=cross, node_radius=radius,
        terms=dict(foreground=case["foreground"], feature=case["features"] > 0, cross_view=cross.count > 0,
                   density=case["density"]),
        surfel_position=surfels, surfel_normal=normals)
    if case["pairs"] and case["features"]:
        scene = synth.with_feature_pairs(scene, per_view=case["features"], seed=seed)
    return scene


def _batch_scenes(case, seed):
    """Scenes of a batch: node counts (and views) spread over the range, or
    initial fields of one subject where every member has the same size."""
    if case["min_nodes"] >= case["nodes"]:
        base = _scene(case, seed)
        return [base] + [synth.perturb_warp_field(base, seed=seed * 1000 + k) for k in range(1, case["count"])]
    out = []
    for k in range(case["count"]):
        n = case["min_nodes"] * (case["nodes"] / case["min_nodes"]) ** (k / max(1, case["count"] - 1))
        out.append(_scene(case, seed * 1000 + k, nodes=int(n), views=1 + (k * 5 + 2) % case["views"]))
    return out


def _config(case, scene, **more):
    return abi.make_config(
        scene, precision=abi.PRECISION_MIXED if case["precision"] == "mixed" else abi.PRECISION_FP32,
        mode=abi.MODE_MATERIALIZED if case["mode"] == "materialized" else abi.MODE_MATRIX_FREE,
        num_global_iterations=case["global_iterations"], **more)


def _surfel_cloud(case, seed):
    """Surfels on a warped sheet with their skinning and field (GPU tensors)."""
    gen = torch.Generator(DEV)
    gen.manual_seed(int(np.random.default_rng(seed).integers(1 << 60)))
    S, N = case["surfels"], case["nodes"]

    def points(n):
        a = torch.rand((n, 2), generator=gen, device=DEV, dtype=F64)
        th, h = 2 * math.pi * a[:, 0], 1.2 * a[:, 1] - 0.6
        n3 = torch.stack([torch.sin(th), 0.2 * torch.sin(9 * h), torch.cos(th)], 1)
        return torch.stack([0.25 * torch.sin(th), h, 0.15 * torch.cos(th) + 1.3], 1), n3 / n3.norm(dim=1, keepdim=True)

    p, n = points(S)
    # surfels are stored in the scan order of the views that added them
    order = torch.argsort(torch.floor(p[:, 1] * 400).to(torch.int64) * 4096 + torch.floor(p[:, 0] * 4000).to(torch.int64))
    p, n = p[order], n[order]
    nodes, _ = points(N)
    knn, w = _skin(p, nodes, 0.025)
    nk, nw = _skin(nodes, nodes, 0.025)
    f32 = torch.float32
    conf = torch.rand((S, 1), generator=gen, device=DEV, dtype=F64)

    def cat(x, tail):
        return torch.cat([x, tail], 1).to(f32).contiguous()

    def u16(x):
        return x.to(torch.int32).to(torch.int16).contiguous()  # the low 16 bits

    # a per-surfel rigid correction that the inverse warp undoes
    d = torch.randn((S, 3), generator=gen, device=DEV, dtype=F64) * 0.01
    c, s = torch.cos(d[:, 0]), torch.sin(d[:, 0])
    z, o = torch.zeros_like(c), torch.ones_like(c)
    correct = torch.cat([torch.stack([c, s, z, -s, c, z, z, z, o], 1), d], 1).to(f32).contiguous()
    return dict(field=torch.from_numpy(_warp_field(nodes, gen)).to(DEV), knn=u16(knn), w=w.to(f32).contiguous(),
                v=cat(p, 20 * conf), n=cat(n, conf), node_knn=u16(nk), node_w=nw.to(f32).contiguous(),
                nodes=cat(nodes, torch.ones((N, 1), dtype=F64, device=DEV)), correct=correct)


def _matrix(case, seed):
    """A block-CSR matrix with a diagonal block and 1 .. 2 per_row - 1 further
    blocks in each row, and a vector (GPU tensors)."""
    gen = torch.Generator(DEV)
    gen.manual_seed(int(np.random.default_rng(seed).integers(1 << 60)))
    n = case["rows"]
    count = torch.randint(2, 2 * case["per_row"], (n,), generator=gen, device=DEV)
    rowptr = torch.cat([count.new_zeros(1), count.cumsum(0)])
    nnz = int(rowptr[-1])
    row = torch.arange(n, device=DEV).repeat_interleave(count)
    near = row + torch.round(torch.randn(nnz, generator=gen, device=DEV, dtype=F64) * n * 0.1).to(torch.int64)
    col = near.remainder(n)
    col[rowptr[:-1]] = torch.arange(n, device=DEV)
    blocks = torch.randn((nnz, 36), generator=gen, device=DEV, dtype=torch.float32)
    x = torch.randn(6 * n, generator=gen, device=DEV, dtype=torch.float32)
    return dict(rowptr=rowptr.to(torch.int32), col=col.to(torch.int32), blocks=blocks, x=x)


# ------------------------------------------------------------ prepare, run ----

def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        scene = _scene(case, seed)
        solver = NonRigidSolver(_config(case, scene))
        return dict(case=case, solver=solver, inputs=DeviceScene(scene, density=case["density"]))
    if kind == "batch":
        scenes = _batch_scenes(case, seed)
        cfg = _config(case, None, max_nodes=max(s.num_nodes for s in scenes), max_views=case["views"],
                      width=case["width"], height=case["height"], max_surfels=max(s.num_surfels for s in scenes),
                      use_foreground=case["foreground"], use_feature=case["features"] > 0,
                      use_cross_view=case["cross"] > 0, max_feature_terms=max(s.feature.count for s in scenes),
                      max_cross_terms=max(s.cross_view.count for s in scenes))
        batch = StreamedBatch(cfg, case["count"], lanes=2)
        state = dict(case=case, batch=batch, inputs=[DeviceScene(s) for s in scenes],
                     out=[torch.empty((s.num_nodes, 8), dtype=torch.float32, device=DEV) for s in scenes])
        # a program tunes and captures its batch once and then feeds it
        for i, ds in enumerate(state["inputs"]):
            batch.set_input(i, ds)
        batch.autotune()
        run(state)
        return state
    if kind == "warp":
        return dict(case=case, **_surfel_cloud(case, seed))
    if kind == "node_error":
        scene = _scene(case, seed)
        solver = NonRigidSolver(_config(case, scene))
        solver.set_solver_input(scene)
        return dict(case=case, solver=solver)
    if kind == "solver_maps":
        scene = _scene(case, seed)
        return dict(case=case, geometry=_geometry(scene, seed), cameras=scene.views, renderer=SolverMapRenderer(
            case["width"], case["height"], case["views"], sized_view0=case["sized"]))
    m = _matrix(case, seed)
    m.update(case=case, y=torch.empty_like(m["x"]), dot=torch.empty(1, dtype=F64, device=DEV))
    return m


def _geometry(scene, seed):
    """The renderer's surfel arrays (GPU tensors), moved by the scene's field."""
    gen = torch.Generator(DEV)
    gen.manual_seed(int(np.random.default_rng([seed, 17]).integers(1 << 60)))
    p, n = scene.surfel_position, scene.surfel_normal
    S = len(p)

    def uniform(lo, hi):
        return lo + (hi - lo) * torch.rand((S, 1), generator=gen, device=DEV, dtype=F64)

    q, t = _blend(_dq(scene.node_se3), torch.from_numpy(scene.surfel_knn.astype(np.int64)).to(DEV),
                  torch.from_numpy(scene.surfel_knn_weight).to(DEV, F64))
    m = np.asarray(scene.views[0].initial_camera_se3, np.float64)
    axis = torch.as_tensor(m[6:9], device=DEV)  # the camera's z axis
    depth = ((p - torch.as_tensor(m[9:], device=DEV)) @ axis).abs()[:, None]
    radius = depth / float(scene.views[0].intrinsic[2]) * 1000.0 * uniform(0.5, 1.5)
    conf = uniform(0.0, 20.0)
    rgb = torch.randint(0, 1 << 24, (S, 1), generator=gen, device=DEV, dtype=torch.int32).view(torch.float32)
    seen = torch.floor(uniform(4.0, 10.99)).to(torch.float32)
    born = torch.floor(uniform(0.0, 10.99)).to(torch.float32)

    def cat(x, tail):
        return torch.cat([x, tail], 1).to(torch.float32).contiguous()

    return dict(reference_vertex_confid=cat(p, conf), reference_normal_radius=cat(n, radius),
                live_vertex_confid=cat(_rotate(q, p) + t, conf), live_normal_radius=cat(_rotate(q, n), radius),
                color_time=torch.cat([rgb, born, seen, torch.zeros_like(seen)], 1).contiguous())


def run(state):
    kind = state["case"]["kind"]
    if kind == "frame":
        solver = state["solver"]
        solver.set_solver_input(state["inputs"])
        solver.solve_non_rigid_alignment(state["case"]["gn"], state["case"]["pcg"])
        return solver.solved_node_se3()
    if kind == "batch":
        batch = state["batch"]
        for i, ds in enumerate(state["inputs"]):
            batch.set_input(i, ds)
        batch.solve(state["case"]["gn"], state["case"]["pcg"])
        return [batch.node_se3_async(i, o) for i, o in enumerate(state["out"])]
    if kind == "warp":
        s = state
        lv, ln, nodes = SurfelNodeDeformer.forward_warp_surfels_and_nodes(
            s["field"], s["knn"], s["w"], s["v"], s["n"], s["node_knn"], s["node_w"], s["nodes"])
        rv, rn = SurfelNodeDeformer.inverse_warp_surfels(s["field"], s["knn"], s["w"], lv, ln, s["correct"])
        return [lv, ln, nodes, rv, rn]
    if kind == "node_error":
        return state["solver"].compute_alignment_error_on_nodes(maps=True)
    if kind == "solver_maps":
        r = state["renderer"]
        r.draw_solver_maps_with_recent_observation(state["geometry"], 10.0, state["cameras"])
        return [r.reference_vertex, r.reference_normal, r.live_vertex, r.live_normal, r.normalized_rgb, r.index]
    s = state
    stream = torch.cuda.current_stream().cuda_stream
    check(lib().mvdr_bsr6_spmv_dot_noalloc(
        s["case"]["rows"], len(s["blocks"]), s["rowptr"].data_ptr(), s["col"].data_ptr(), s["blocks"].data_ptr(),
        s["x"].data_ptr(), s["y"].data_ptr(), s["dot"].data_ptr(), C.c_void_p(stream)))
    return [s["y"], s["dot"]]


def work(case):
    """Inputs read once, outputs written once; the arithmetic of one pass."""
    kind = case["kind"]
    if kind == "warp":
        S, N = case["surfels"], case["nodes"]
        return dict(bytes=S * (8 + 16 + 32 + 32) + N * 56 + S * (48 + 32), flops=S * 2 * 190)
    if kind == "spmv":
        nnz = case["rows"] * case["per_row"]
        return dict(bytes=nnz * 148 + case["rows"] * 52, flops=nnz * 72)
    pixels = case["views"] * case["width"] * case["height"]
    drawn = pixels * _coverage(case)
    if kind == "node_error":
        return dict(bytes=pixels * 12 + drawn * (32 + 24 + 36) + case["nodes"] * 48, flops=drawn * 500)
    if kind == "solver_maps":
        return dict(bytes=pixels * 84 + drawn * 80, flops=drawn * (60 * case["views"] + 100))
    scale, nodes, views = 1.0, case["nodes"], case["views"]
    if kind == "batch" and case["min_nodes"] < nodes:  # the mean of a spread batch
        nodes, scale = math.sqrt(nodes * case["min_nodes"]) * 1.2, 0.5 + 0.5 / views
    scale *= case.get("count", 1)
    terms = (2.2 if case["density"] else 1.2 if case["foreground"] else 1.0) * drawn
    per_pixel = 68 + (12 if case["foreground"] else 0) + (28 if case["density"] else 0)
    nbytes = pixels * per_pixel + drawn * 24 + nodes * (64 + 32) + 56 * views * (case["features"] + case["cross"])
    # per iteration: 150 operations a term, 42 for each of its ten blocks; a
    # product with about 20 blocks a row in each PCG iteration
    flops = case["gn"] * (terms * (150 + 420) + case["pcg"] * nodes * 20 * 72)
    return dict(bytes=scale * nbytes, flops=scale * flops)


# ------------------------------------------------- the same in 64 bits --------

def _dq(field):
    return torch.as_tensor(field).to(DEV, F64)


def _qmul(a, b):
    ax, ay, az, aw = a.unbind(-1)
    bx, by, bz, bw = b.unbind(-1)
    return torch.stack([aw * bx + ax * bw + ay * bz - az * by, aw * by - ax * bz + ay * bw + az * bx,
                        aw * bz + ax * by - ay * bx + az * bw, aw * bw - ax * bx - ay * by - az * bz], -1)


def _rigid(dq):
    """Unit rotation quaternion and translation of dual quaternions."""
    inv = dq[:, :4].norm(dim=1, keepdim=True).reciprocal()
    q0, q1 = dq[:, :4] * inv, dq[:, 4:] * inv
    q1 = q1 - (q0 * q1).sum(1, keepdim=True) * q0
    conj = q0 * q0.new_tensor([-1.0, -1.0, -1.0, 1.0])
    return q0, _qmul(2 * q1, conj)[:, :3]


def _blend(dq, knn, w):
    return _rigid((dq[knn] * w[:, :, None]).sum(1))


def _rotate(q, p):
    v, s = q[:, :3], q[:, 3:]
    u = torch.linalg.cross(v, p)
    return p + 2 * (s * u + torch.linalg.cross(v, u))


def _quat_matrix(q):
    x, y, z, w = q.unbind(-1)
    return torch.stack([1 - 2 * y * y - 2 * z * z, 2 * x * y - 2 * z * w, 2 * x * z + 2 * y * w,
                        2 * x * y + 2 * z * w, 1 - 2 * x * x - 2 * z * z, 2 * y * z - 2 * x * w,
                        2 * x * z - 2 * y * w, 2 * y * z + 2 * x * w, 1 - 2 * x * x - 2 * y * y], -1).reshape(-1, 3, 3)


def _matrix_quat(R):
    m = R.reshape(-1, 9)
    t = [m[:, 0] + m[:, 4] + m[:, 8], m[:, 0] - m[:, 4] - m[:, 8], m[:, 4] - m[:, 0] - m[:, 8], m[:, 8] - m[:, 0] - m[:, 4]]
    d = [m[:, 7] - m[:, 5], m[:, 2] - m[:, 6], m[:, 3] - m[:, 1]]
    s = [m[:, 1] + m[:, 3], m[:, 2] + m[:, 6], m[:, 5] + m[:, 7]]
    forms = []
    for k, rows in enumerate(([d[0], d[1], d[2], None], [None, s[0], s[1], d[0]], [s[0], None, s[2], d[1]],
                              [s[1], s[2], None, d[2]])):
        r = 2 * (1 + t[k]).clamp(min=1e-30).sqrt()
        forms.append(torch.stack([0.25 * r if x is None else x / r for x in rows], 1))
    pick = torch.where(t[0] > 0, 0, torch.where((m[:, 0] > m[:, 4]) & (m[:, 0] > m[:, 8]), 1,
                                                torch.where(m[:, 4] > m[:, 8], 2, 3)))
    return torch.stack(forms, 1)[torch.arange(len(m), device=m.device), pick]


class _Camera:
    def __init__(self, view):
        def mat(a):
            a = torch.as_tensor(np.asarray(a, np.float64), device=DEV)
            return a[:9].reshape(3, 3).T, a[9:]

        self.Rw, self.tw = mat(view.world2camera)
        self.Ri, self.ti = mat(view.initial_camera_se3)
        self.cx, self.cy, self.fx, self.fy = (float(x) for x in view.intrinsic)

    def to_frame0(self, p):
        return p @ self.Ri.T + self.ti

    def to_camera(self, p):
        return (p @ self.Rw.T + self.tw - self.ti) @ self.Ri

    def turn(self, n):  # frame 0 -> camera, directions
        return n @ self.Rw.T @ self.Ri

    def turn_back(self, n):
        return n @ self.Ri.T @ self.Rw

    def pixel(self, p):
        z = p[:, 2] + 1e-10
        return (torch.round((p[:, 0] / z * self.fx + self.cx).float()).to(torch.int64),
                torch.round((p[:, 1] / z * self.fy + self.cy).float()).to(torch.int64))


def _map(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV, F64)


def _image_rows(cam, gradient, vc, wv, p):
    """Twist gradient of an image sampled at the projection of vc."""
    gr = gradient.reshape(-1, 2)[p]
    z = vc[:, 2]
    g = torch.stack([gr[:, 0] * cam.fx / z, gr[:, 1] * cam.fy / z,
                     -(cam.fx * vc[:, 0] * gr[:, 0] + cam.fy * vc[:, 1] * gr[:, 1]) / (z * z)], 1)
    g = cam.turn_back(g)
    return torch.cat([torch.linalg.cross(wv, g), g], 1)


def _twist_rows(p):
    """[p]x^T | I: the three Jacobian rows of a moved point (n, 3, 6)."""
    z = torch.zeros_like(p[:, 0])
    x, y, c = p.unbind(-1)
    skew = torch.stack([z, c, -y, -c, z, x, y, -x, z], -1).reshape(-1, 3, 3)
    return torch.cat([skew, torch.eye(3, dtype=F64, device=DEV).expand(len(p), 3, 3)], 2)


class _Rows:
    """Weighted Jacobian rows: row t has nodes[t, k] with gradient J[t, k]
    (or w[t, k] times one J[t]) and residual r[t]."""

    def __init__(self, nodes, w, J, r):
        self.nodes, self.w, self.J, self.r = nodes, w, J, r

    def parts(self, k):
        return self.J * self.w[:, k, None] if self.J.dim() == 2 else self.J[:, k]

    def dot(self, d):
        if self.J.dim() == 2:
            return ((d[self.nodes] * self.w[:, :, None]).sum(1) * self.J).sum(1)
        return (d[self.nodes] * self.J).sum((1, 2))

    def transposed(self, y, out):
        for k in range(self.nodes.shape[1]):
            out.index_add_(0, self.nodes[:, k], self.parts(k) * y[:, None])


class _Solve:
    """The Gauss-Newton solve of one scene in float64."""

    def __init__(self, case, scene):
        self.case, self.scene, self.N = case, scene, scene.num_nodes
        self.dq = _dq(scene.node_se3)
        self.cams = [_Camera(v) for v in scene.views]
        self.knn = torch.from_numpy(scene.surfel_knn.astype(np.int64)).to(DEV)
        self.w = _map(scene.surfel_knn_weight)
        self.nodes = _map(scene.canonical_nodes)[:, :3]
        self.edges = torch.from_numpy(scene.node_graph.astype(np.int64)).to(DEV)
        self.H, self.W = scene.height, scene.width
        self.pixels = []
        for cam, v in zip(self.cams, scene.views):
            idx = torch.from_numpy(v.index_map.astype(np.int64)).to(DEV).reshape(-1)
            pix = (idx != EMPTY).nonzero()[:, 0]
            rv, rn = (_map(a).reshape(-1, 4)[pix, :3] for a in (v.reference_vertex_map, v.reference_normal_map))
            e = dict(pix=pix, s=idx[pix], p=cam.to_frame0(rv), n=rn @ cam.Ri.T, obs_v=_map(v.vertex_confidence_map),
                     obs_n=_map(v.normal_radius_map), fg=_map(v.filtered_foreground_mask),
                     fg_grad=_map(v.foreground_mask_gradient))
            if case["density"]:
                rgb = _map(v.normalized_rgb_map).reshape(-1, 4)[pix]
                e.update(grey=rgb[:, :3] @ rgb.new_tensor([0.299, 0.587, 0.114]), dens=_map(v.density_map).reshape(-1),
                         dens_grad=_map(v.density_gradient_map))
            if case["foreground"]:
                wv, vc, nc = self.moved(cam, e)
                p, ok = self.inside(cam, vc)
                ok &= -(vc * nc).sum(1) / vc.norm(dim=1) > 0.5
                e["fg_terms"] = ok & (e["fg"].reshape(-1)[p] > 1e-5)
            self.pixels.append(e)
        self.points = []
        if case["features"]:
            self.points.append(("feature", *(self.selected() if scene.feature_pairs else self.given(scene.feature))))
        if scene.cross_view.count:
            self.points.append(("cross", *self.given(scene.cross_view)))

    @staticmethod
    def given(c):
        return (torch.from_numpy(c.knn.astype(np.int64)).to(DEV), _map(c.knn_weight),
                _map(c.reference_vertex)[:, :3], _map(c.target_vertex)[:, :3])

    def selected(self):
        """The feature terms of raw pixel pairs: the observed pixel is the
        pair's (or a neighbour with a depth), the rendered one the nearest of
        its 3x3 window."""
        got = []
        for cam, view, e, (pairs, live, edge) in zip(self.cams, self.scene.views, self.pixels, self.scene.feature_pairs):
            q = torch.from_numpy(pairs.astype(np.int64)).to(DEV)
            obs, ref, live = e["obs_v"][..., :3], _map(view.reference_vertex_map)[..., :3], _map(live)[..., :3]
            idx = torch.from_numpy(view.index_map.astype(np.int64)).to(DEV)
            edge = torch.from_numpy(edge).to(DEV)

            def at(m, x, y, fill):
                ok = (x >= 0) & (y >= 0) & (x < self.W) & (y < self.H)
                v = m[y.clamp(0, self.H - 1), x.clamp(0, self.W - 1)]
                return torch.where(ok[:, None] if v.dim() == 2 else ok, v, torch.full_like(v, fill)), ok

            def real(x, y):
                return ~(at(obs, x, y, 0.0)[0].abs() < 1e-3).all(1)

            dx, dy = torch.full_like(q[:, 0], -1), torch.full_like(q[:, 0], -1)
            for j in (-1, 0, 1):
                for i in (1, 0, -1):  # the last row's first pixel with a depth
                    x, y = q[:, 2] + i, q[:, 3] + j
                    ok = real(x, y)
                    dx, dy = torch.where(ok, x, dx), torch.where(ok, y, dy)
            ok = real(q[:, 2], q[:, 3])
            dx, dy = torch.where(ok, q[:, 2], dx), torch.where(ok, q[:, 3], dy)
            keep = (dx >= 0) & (dy >= 0) & (dx < self.W) & (dy < self.H)
            ov = at(obs, dx, dy, 0.0)[0]
            keep &= at(edge, dx, dy, 0)[0] != 1
            best = torch.full((len(q),), 100.0, dtype=F64, device=DEV)
            gx, gy = torch.full_like(dx, -1), torch.full_like(dx, -1)
            for j in (-1, 0, 1):
                for i in (-1, 0, 1):
                    x, y = q[:, 0] + i, q[:, 1] + j
                    d = ((ov - at(live, x, y, 0.0)[0]) ** 2).sum(1)
                    ok = (at(idx, x, y, 0)[0] != EMPTY) & (d < best)
                    best, gx, gy = torch.where(ok, d, best), torch.where(ok, x, gx), torch.where(ok, y, gy)
            keep &= (gx >= 0) & (gy >= 0) & (gx < self.W) & (gy < self.H)
            s = at(idx, gx, gy, EMPTY)[0]
            rv = at(ref, gx, gy, 0.0)[0]
            keep &= (s < self.scene.num_surfels) & (((rv - ov) ** 2).sum(1) < 2.5e-3)
            s, rv, ov = s[keep], rv[keep], ov[keep]
            got.append((self.knn[s], self.w[s], cam.to_frame0(rv), (cam.to_frame0(ov) - cam.tw) @ cam.Rw))
        return tuple(torch.cat(x) for x in zip(*got))

    def moved(self, cam, e, keep=slice(None)):
        q, t = _blend(self.dq, self.knn[e["s"][keep]], self.w[e["s"][keep]])
        wv = _rotate(q, e["p"][keep]) + t
        return wv, cam.to_camera(wv), cam.turn(_rotate(q, e["n"][keep]))

    def inside(self, cam, vc):
        x, y = cam.pixel(vc)
        ok = (x >= 0) & (x < self.W) & (y >= 0) & (y < self.H)
        return torch.where(ok, y * self.W + x, 0), ok

    def rows(self, it):
        local = it >= self.case["global_iterations"]
        smooth, density, fg = 5.0, float(np.float32(1e-2)) if local else 0.0, 0.0 if local else float(np.float32(2e-3))
        lam = dict(feature=0.0 if local else 1.0, cross=1.0)
        out = []
        for cam, e in zip(self.cams, self.pixels):
            wv, vc, nc = self.moved(cam, e)
            p, ok = self.inside(cam, vc)
            dv, dn = e["obs_v"].reshape(-1, 4)[p, :3], e["obs_n"].reshape(-1, 4)[p, :3]
            dense = ok & ~(dv.abs() < 1e-3).all(1) & ((dn * nc).sum(1) >= float(np.float32(0.7)))
            dense &= ((dv - vc) ** 2).sum(1) <= float(np.float32(0.075) * np.float32(0.075))
            back = cam.turn_back(dn[dense])
            s = e["s"][dense]
            out.append(_Rows(self.knn[s], self.w[s], torch.cat([torch.linalg.cross(wv[dense], back), back], 1),
                             (dn * (vc - dv)).sum(1)[dense]))
            for on, lam_i, grad, image in ((ok, density, "dens_grad", "dens"), (e.get("fg_terms"), fg, "fg_grad", "fg")):
                if lam_i == 0.0 or grad not in e or on is None:
                    continue
                on = on & ok
                s = e["s"][on]
                J = _image_rows(cam, e[grad], vc[on], wv[on], p[on])
                r = e[image].reshape(-1)[p[on]] - (e["grey"][on] if image == "dens" else 0.0)
                out.append(_Rows(self.knn[s], self.w[s], lam_i * J, lam_i * r))
        q, t = _rigid(self.dq)
        i, j = self.edges.unbind(1)
        near = ((self.nodes[i] - self.nodes[j]) ** 2).sum(1) <= 64.0 * self.scene.node_radius ** 2
        i, j = i[near], j[near]
        a, b = _rotate(q[i], self.nodes[j]) + t[i], _rotate(q[j], self.nodes[j]) + t[j]
        J = torch.stack([_twist_rows(a), -_twist_rows(b)], 2).reshape(-1, 2, 6)
        out.append(_Rows(torch.stack([i, j], 1).repeat_interleave(3, 0), None, smooth * J, smooth * (a - b).reshape(-1)))
        for name, knn, w, ref, tgt in self.points:
            if lam[name] == 0.0:
                continue
            q, t = _blend(self.dq, knn, w)
            wv = _rotate(q, ref) + t
            raw = wv - tgt
            cut = float(np.float32(7.5e-2))
            hub = torch.where(raw.abs() < cut, torch.ones_like(raw), cut / raw.abs())
            J = (lam[name] * hub[:, :, None] * _twist_rows(wv)).reshape(-1, 6)
            out.append(_Rows(knn.repeat_interleave(3, 0), w.repeat_interleave(3, 0), J, lam[name] * (hub * raw).reshape(-1)))
        return out

    def iterate(self, it):
        rows = self.rows(it)
        damp = float(np.float32(1e-2))
        b = torch.zeros((self.N, 6), dtype=F64, device=DEV)
        D = torch.zeros((self.N, 36), dtype=F64, device=DEV)
        for g in rows:
            g.transposed(-g.r, b)
            for k in range(g.nodes.shape[1]):
                J = g.parts(k)
                D.index_add_(0, g.nodes[:, k], (J[:, :, None] * J[:, None, :]).reshape(-1, 36))
        L = torch.linalg.cholesky(D.reshape(-1, 6, 6) + damp * torch.eye(6, dtype=F64, device=DEV))

        def apply(d):
            y = damp * d
            for g in rows:
                g.transposed(g.dot(d), y)
            return y

        def precondition(v):
            return torch.cholesky_solve(v[:, :, None], L)[:, :, 0]

        x, r = torch.zeros_like(b), b.clone()
        s = precondition(r)
        d, delta = s, (r * s).sum()
        for _ in range(self.case["pcg"]):
            q = apply(d)
            alpha = delta / (d * q).sum()
            x, r = x + alpha * d, r - alpha * q
            s = precondition(r)
            new = (r * s).sum()
            d, delta = s + new / delta * d, new
        om, tr = x[:, :3], x[:, 3:]
        ang = om.norm(dim=1, keepdim=True).clamp(min=1e-30)
        ax = om / ang
        K = -_twist_rows(ax)[:, :, :3]
        R = torch.eye(3, dtype=F64, device=DEV) + torch.sin(ang)[:, :, None] * K + (1 - torch.cos(ang))[:, :, None] * (K @ K)
        R = torch.where((om.abs().sum(1) < 1e-4)[:, None, None], torch.eye(3, dtype=F64, device=DEV), R)
        q, t = _rigid(self.dq)
        q0 = _matrix_quat(R @ _quat_matrix(q))
        t = (R @ t[:, :, None])[:, :, 0] + tr
        self.dq = torch.cat([q0, _qmul(torch.cat([0.5 * t, torch.zeros_like(t[:, :1])], 1), q0)], 1)

    def solved(self):
        for it in range(self.case["gn"]):
            self.iterate(it)
        return self.dq


def _exact_warp(case, seed):
    s = _surfel_cloud(case, seed)
    dq = s["field"].to(F64)

    def moved(knn, w):
        return _blend(dq, knn.to(torch.int64) & 0xFFFF, w.to(F64))

    q, t = moved(s["knn"], s["w"])
    v, n = s["v"].to(F64), s["n"].to(F64)
    lv = torch.cat([_rotate(q, v[:, :3]) + t, v[:, 3:]], 1)
    ln = torch.cat([_rotate(q, n[:, :3]), n[:, 3:]], 1)
    qn, tn = moved(s["node_knn"], s["node_w"])
    nodes = s["nodes"].to(F64)
    live_nodes = torch.cat([_rotate(qn, nodes[:, :3]) + tn, nodes[:, 3:]], 1)
    # the inverse warp undoes the field, then the correction (whose rotation's
    # inverse is its transpose)
    c = s["correct"].to(F64)
    Rc = c[:, :9].reshape(-1, 3, 3)  # rotation columns: already transposed
    p = (Rc @ (v[:, :3] - c[:, 9:])[:, :, None])[:, :, 0]
    m = (Rc @ n[:, :3, None])[:, :, 0]
    return [lv, ln, live_nodes, torch.cat([p, v[:, 3:]], 1), torch.cat([m, n[:, 3:]], 1)]


def _exact_node_error(case, seed):
    s = _Solve(dict(case, foreground=False), _scene(case, seed))
    H, W, N = s.H, s.W, s.N
    err = torch.zeros((len(s.cams), H * W), dtype=F64, device=DEV)
    acc, weight = torch.zeros(N, dtype=F64, device=DEV), torch.zeros(N, dtype=F64, device=DEV)
    for v, (cam, e) in enumerate(zip(s.cams, s.pixels)):
        _, vc, nc = s.moved(cam, e)
        x, y = cam.pixel(vc)
        x, y = x.clamp(-2, W + 1), y.clamp(-2, H + 1)
        best = torch.full_like(vc[:, 0], float(np.float32(0.1)))
        found = torch.zeros_like(best, dtype=torch.bool)
        for j in (-1, 0, 1):
            for i in (-1, 0, 1):
                ok = (x + i >= 0) & (x + i < W) & (y + j >= 0) & (y + j < H)
                p = torch.where(ok, (y + j) * W + x + i, 0)
                dv, dn = (torch.where(ok[:, None], e[m].reshape(-1, 4)[p, :3], 0.0) for m in ("obs_v", "obs_n"))
                found |= ~(dv.abs() < 1e-3).all(1) & ((nc * dn).sum(1) > float(np.float32(0.7)))
                best = torch.minimum(best, (vc - dv).abs().sum(1))
        ok = (x >= 0) & (x < W) & (y >= 0) & (y < H)
        fg = torch.where(ok, e["fg"].reshape(-1)[torch.where(ok, y * W + x, 0)], 0.0)
        best = torch.where(found, best, torch.where(fg < 0.9, 0.03 * fg, float(np.float32(0.1))))
        err[v, e["pix"]] = best
        on = best > 1e-6
        k, w = s.knn[e["s"][on]], s.w[e["s"][on]]
        acc.index_add_(0, k.reshape(-1), (w * best[on, None]).reshape(-1))
        weight.index_add_(0, k.reshape(-1), w.reshape(-1))
    united = torch.where(acc < 1e-10, torch.ones_like(acc), acc / (weight + 1e-4) / float(np.float32(0.1)))
    back = torch.zeros_like(err)
    for v, e in enumerate(s.pixels):
        k, w = s.knn[e["s"]], s.w[e["s"]]
        back[v, e["pix"]] = ((acc / weight)[k] * w).sum(1) / (w.sum(1) + 1e-4)
    shape = (len(s.cams), H, W)
    return dict(accumulated_error=acc, accumulated_weight=weight, united_error=united, large_error_mark=None,
                alignment_error_map=err.reshape(shape), node_error_map=back.reshape(shape))


def _exact_solver_maps(case, seed):
    scene = _scene(case, seed)
    g = {k: v.to(F64) for k, v in _geometry(scene, seed).items()}
    bits = _geometry(scene, seed)["color_time"][:, 0].contiguous().view(torch.int32).to(torch.int64)
    H, W = case["height"], case["width"]
    live, conf = g["live_vertex_confid"][:, :3], g["reference_vertex_confid"][:, 3]
    shown = (conf >= 10.0) | ((g["color_time"][:, 2] - 10.0).abs() < 3.0)
    out = [[] for _ in range(5)]
    for v, view in enumerate(scene.views):
        cam, sized = _Camera(view), case["sized"] and v == 0

        def local(p):
            return (p - cam.ti) @ cam.Ri

        pc = local(live) @ cam.Rw.T + cam.tw
        z = pc[:, 2]

        def image(p):
            return cam.fx * p[:, 0] / p[:, 2] + cam.cx, cam.fy * p[:, 1] / p[:, 2] + cam.cy

        x, y = image(pc)
        ids = (shown & (z > 0) & (z <= 3.05) & (x >= 0) & (x <= W) & (y >= 0) & (y <= H)).nonzero()[:, 0]
        pc, z, x, y = pc[ids], z[ids], x[ids], y[ids]
        size = torch.ones_like(z)
        if sized:
            n = g["live_normal_radius"][ids, :3] @ cam.Ri @ cam.Rw.T
            n = n / n.norm(dim=1, keepdim=True)
            a = torch.stack([n[:, 1] - n[:, 2], -n[:, 0], n[:, 0]], 1)
            a = a / a.norm(dim=1, keepdim=True) * (g["live_normal_radius"][ids, 3:] * 1.41421356 * 0.001)
            b = torch.linalg.cross(n, a)
            p = [image(pc + s * o) for o in (a, b) for s in (1, -1)]
            ext = [torch.stack(c).amax(0) - torch.stack(c).amin(0) for c in zip(*p)]
            size = torch.minimum(*ext).clamp(1.0, 2047.0)
        h = 0.5 * size
        u0, u1 = torch.ceil(x - h - 0.5).clamp(min=0), torch.ceil(x + h - 0.5).clamp(max=W)
        w0, w1 = torch.ceil(y - h - 0.5).clamp(min=0), torch.ceil(y + h - 0.5).clamp(max=H)
        depth = torch.full((H * W,), math.inf, dtype=F64, device=DEV)
        win = torch.full((H * W,), len(live), dtype=torch.int64, device=DEV)
        reach = int(max((u1 - u0).max(), (w1 - w0).max()))
        spots = []
        for j in range(reach):
            for i in range(reach):
                on = ((u0 + i < u1) & (w0 + j < w1)).nonzero()[:, 0]
                pix = ((w0[on] + j) * W + u0[on] + i).to(torch.int64)
                depth.scatter_reduce_(0, pix, z[on], "amin")
                spots.append((on, pix))
        for on, pix in spots:
            near = z[on] == depth[pix]
            win.scatter_reduce_(0, pix[near], ids[on[near]], "amin")
        hit = (win < len(live)).nonzero()[:, 0]
        s = win[hit]
        for k, (name, point) in enumerate((("reference_vertex_confid", True), ("reference_normal_radius", False),
                                           ("live_vertex_confid", True), ("live_normal_radius", False))):
            m = torch.zeros((H * W, 4), dtype=F64, device=DEV)
            a = g[name][s, :3]
            m[hit, :3] = local(a) if point else a @ cam.Ri
            m[hit, 3] = 1.0 if point else 0.0
            out[k].append(m.reshape(H, W, 4))
        m = torch.zeros((H * W, 4), dtype=F64, device=DEV)
        for c in range(3):
            m[hit, c] = ((bits[s] >> (16 - 8 * c)) & 255).to(F64) / 255.0
        m[hit, 3] = 1.0 if sized else g["color_time"][s, 1]
        out[4].append(m.reshape(H, W, 4))
    return [torch.stack(x) for x in out] + [None]


def exact(case, seed):
    kind = case["kind"]
    if kind == "frame":
        return _Solve(case, _scene(case, seed)).solved()
    if kind == "batch":
        return [_Solve(case, s).solved() for s in _batch_scenes(case, seed)]
    if kind == "warp":
        return _exact_warp(case, seed)
    if kind == "node_error":
        return _exact_node_error(case, seed)
    if kind == "solver_maps":
        return _exact_solver_maps(case, seed)
    m = _matrix(case, seed)
    n = case["rows"]
    row = torch.arange(n, device=DEV).repeat_interleave((m["rowptr"][1:] - m["rowptr"][:-1]).to(torch.int64))
    x = m["x"].to(F64)
    prod = (m["blocks"].to(F64).reshape(-1, 6, 6) @ x.reshape(n, 6)[m["col"].to(torch.int64)][:, :, None])[:, :, 0]
    y = torch.zeros((n, 6), dtype=F64, device=DEV).index_add_(0, row, prod).reshape(-1)
    # the call's dot product is that of x with the y it returned in float32
    return [y, torch.dot(x, y.to(torch.float32).to(F64))[None]]
