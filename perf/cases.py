"""Performance cases of the normal-estimation path, through the public Python API.

A case is a dict of plain values. `prepare` makes what a caller holds before
the call (point arrays, a context, a trained radius model, a built tree where
the tree is kept), `run` is one pass through the entry points, `work` the bytes
and operations a pass cannot do without, `exact` the same results in 64 bits
where a brute-force search can give them.

Kinds of case:

* ``normals``  cloud in, normals out: ``Context.build`` + ``Context.normals``
               (``mem`` device: torch CUDA tensors; host: the drop-in classes
               ``PointCloud`` -> ``RadixTree`` -> ``Octree`` ->
               ``NormalEstimation.estimateNormals`` on numpy arrays)
* ``lists``    cloud in, neighbour lists and squared distances out:
               ``Context.build`` + ``Context.knn_self``
* ``queries``  neighbours of foreign query points in a kept tree: ``Context.knn``
* ``batch``    many independent clouds in one call: ``Context.normals_batch``
* ``train``    the learned search radius: ``Context.mlp_init`` + ``mlp_train``
"""
from __future__ import annotations

import math

import numpy as np
import torch

from shapeextraction_b200 import Context, NormalEstimation, Octree, PointCloud, RadixTree
from shapeextraction_b200.learned import radius_targets, train_radius_model

EXACT_POINTS = 120_000  # largest cloud the brute-force 64-bit search takes on


def listed():
    return [
        # one scan line, segment or object: latency and launches are everything
        {"name": "object_2k_k8", "kind": "normals", "cloud": "scene", "n": 2_011, "k": 8},
        # the 30-bit configuration: a small unstructured volume
        {"name": "cube_100k_k10_30bit", "kind": "normals", "cloud": "cube", "n": 100_000, "k": 10, "code_bits": 30},
        # the reference's own calling sequence on host arrays, with its default k
        {"name": "classes_host_100k_k8", "kind": "normals", "cloud": "scene", "n": 100_003, "k": 8, "mem": "host"},
        # one LiDAR scene
        {"name": "scene_2M_k16", "kind": "normals", "cloud": "scene", "n": 2_000_000, "k": 16},
        # the same with the learned search radius, model trained beforehand on another cloud
        {"name": "scene_2M_k16_learned", "kind": "normals", "cloud": "scene", "n": 2_000_000, "k": 16,
         "learned": True},
        # the precision workload: surfaces, thin planes, lines, tiny far clusters; FP64 redo below a 1e-6 gap
        {"name": "precision_20M_k16", "kind": "normals", "cloud": "precision", "n": 20_000_000, "k": 16,
         "gap": 1e-6},
        # the largest cloud: strongly varying density
        {"name": "mixture_50M_k16", "kind": "normals", "cloud": "mixture", "n": 50_000_000, "k": 16},
        # neighbour graph of a cloud, no octree wanted, long lists
        {"name": "lists_1M_k32", "kind": "lists", "cloud": "scene", "n": 999_999, "k": 32, "octree": False},
        # registration: points of another scan, in scan order unknown to the tree, against a kept map
        {"name": "queries_250k_in_2M_k8", "kind": "queries", "cloud": "scene", "n": 2_000_000, "queries": 250_001,
         "k": 8},
        # many clouds of very different sizes, k per cloud
        {"name": "batch_256", "kind": "batch", "clouds": 256, "lo": 1_000, "hi": 500_000},
        # callers that need the reference's own approximate neighbour lists
        {"name": "compat_200k_k16", "kind": "normals", "cloud": "scene", "n": 200_000, "k": 16, "compat": True},
        # training of the radius model, a fraction of its usual steps
        {"name": "train_100_steps", "kind": "train", "cloud": "scene", "n": 65_536, "k": 16, "steps": 100,
         "batch": 8_192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["normals", "host", "learned", "compat", "lists", "queries", "batch", "train"],
                       [8, 2, 2, 2, 3, 3, 2, 1])[0]
    cloud = rng.choice(["scene", "cube", "precision", "mixture"])
    if kind == "normals":
        return {"kind": "normals", "cloud": cloud, "n": _log_int(rng, 1_000, 20_000_000), "k": rng.randint(3, 32),
                "code_bits": rng.choice([63, 63, 63, 30]), "octree": rng.random() < 0.7}
    if kind == "host":
        return {"kind": "normals", "cloud": cloud, "n": _log_int(rng, 1_000, 1_000_000), "k": rng.choice([8, 10, 16]),
                "mem": "host"}
    if kind == "learned":
        return {"kind": "normals", "cloud": rng.choice(["scene", "mixture"]), "n": _log_int(rng, 100_000, 8_000_000),
                "k": rng.choice([8, 16, 24]), "learned": True}
    if kind == "compat":
        return {"kind": "normals", "cloud": "scene", "n": _log_int(rng, 2_000, 300_000), "k": rng.choice([8, 10, 16, 32]),
                "compat": True}
    if kind == "lists":
        return {"kind": "lists", "cloud": cloud, "n": _log_int(rng, 1_000, 4_000_000), "k": rng.randint(1, 32),
                "octree": False}
    if kind == "queries":
        return {"kind": "queries", "cloud": cloud, "n": _log_int(rng, 10_000, 4_000_000),
                "queries": _log_int(rng, 100, 1_000_000), "k": rng.randint(1, 32)}
    if kind == "batch":
        return {"kind": "batch", "clouds": rng.randint(4, 256), "lo": 1_000, "hi": _log_int(rng, 10_000, 500_000)}
    return {"kind": "train", "cloud": "scene", "n": _log_int(rng, 20_000, 200_000), "k": rng.choice([8, 16]),
            "steps": rng.randint(50, 200), "batch": rng.choice([1_000, 4_096, 8_192])}


# ---- clouds -----------------------------------------------------------------
# Seeded clouds with the shapes of shapeextraction_b200.synth, made on the GPU.


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rand(g, *shape, lo=0.0, hi=1.0):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _unit(g, n):
    v = _randn(g, n, 3)
    return v / v.norm(dim=1, keepdim=True)


def _planes(g, n, count, sigma):
    """n points on `count` random planes through the unit cube, jittered along the normals by sigma."""
    normal = _unit(g, count)
    center = _rand(g, count, 3, lo=0.2, hi=0.8)
    axis = normal.abs().argmax(1)
    parts, have = [], 0
    while have < n:
        m = 2 * (n - have) + 1024
        i = torch.randint(count, (m,), generator=g, device="cuda")
        p = _rand(g, m, 3)
        nv, ax = normal[i], axis[i].unsqueeze(1)
        along = p.gather(1, ax)
        off = ((p - center[i]) * nv).sum(1, keepdim=True) / nv.gather(1, ax)
        along = along - off  # moves the point onto its plane along the dominant axis
        p.scatter_(1, ax, along)
        keep = ((along >= 0) & (along <= 1)).squeeze(1).nonzero().squeeze(1)[: n - have]
        s = sigma[i[keep]].unsqueeze(1) if torch.is_tensor(sigma) else sigma
        parts.append(p[keep] + _randn(g, keep.numel(), 1) * s * nv[keep])
        have += keep.numel()
    return torch.cat(parts)


def _scene(g, n):
    radius = _rand(g, 32, lo=0.02, hi=0.2)
    center = _rand(g, 32, 3) * (1 - 2 * radius.unsqueeze(1)) + radius.unsqueeze(1)
    area = 4 * math.pi * radius**2
    on_spheres = int(n * float(area.sum() / (area.sum() + 8 * 1.1)))  # a plane cuts about 1.1 out of the cube
    i = torch.multinomial(area, max(on_spheres, 1), replacement=True, generator=g)[:on_spheres]
    r = radius[i].unsqueeze(1) + 0.002 * _randn(g, on_spheres, 1)
    return torch.cat([center[i] + r * _unit(g, on_spheres), _planes(g, n - on_spheres, 8, 0.002)])


def _precision(g, n):
    n_plane, n_line, n_cluster = int(0.25 * n), int(0.15 * n), int(0.2 * n)
    sigma = 10 ** _rand(g, 16, lo=-5, hi=-2)
    a, b = _rand(g, 64, 3), _rand(g, 64, 3)
    i = torch.randint(64, (n_line,), generator=g, device="cuda")
    lines = a[i] + _rand(g, n_line, 1) * (b - a)[i] + 1e-6 * _randn(g, n_line, 3)
    c = 1e3 + _rand(g, 256, 3)
    j = torch.randint(256, (n_cluster,), generator=g, device="cuda")
    return torch.cat([_scene(g, n - n_plane - n_line - n_cluster), _planes(g, n_plane, 16, sigma), lines,
                      c[j] + 1e-4 * _randn(g, n_cluster, 3)])


def _mixture(g, n):
    n_surface = n // 4
    weight = 10 ** _rand(g, 64, lo=0, hi=1.5)
    scale = 10 ** _rand(g, 64, 3, lo=-2.2, hi=-1.0)
    rot = torch.linalg.qr(_randn(g, 64, 3, 3))[0] * scale.unsqueeze(1)
    mean = _rand(g, 64, 3, lo=0.15, hi=0.85)
    # points per component, in proportion to the weights
    edge = (torch.cumsum(weight, 0) / weight.sum() * (n - n_surface)).round().long().tolist()
    parts, first = [_scene(g, n_surface)], 0
    for i, last in enumerate(edge):
        parts.append(mean[i] + _randn(g, last - first, 3) @ rot[i].T)
        first = last
    return torch.cat(parts)


_CLOUDS = {"scene": _scene, "precision": _precision, "mixture": _mixture, "cube": lambda g, n: _rand(g, n, 3)}


def _shuffled(g, p):
    p = p[torch.randperm(p.shape[0], generator=g, device="cuda")].float()
    return [p[:, i].contiguous() for i in range(3)]


def _cloud(case, seed):
    g = _generator(seed)
    return _shuffled(g, _CLOUDS[case["cloud"]](g, case["n"]))


# ---- what a caller holds before the call ------------------------------------


def _context(case):
    return Context(code_bits=case.get("code_bits", 63), build_octree=case.get("octree", True),
                   eigengap_fp64=case.get("gap", 1e-4), search_compat=case.get("compat", False))


def prepare(case, seed):
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    xyz = _cloud(case, seed)
    ctx = _context(case)
    n, k = case["n"], case["k"]
    state = {"case": case, "ctx": ctx, "xyz": xyz}
    if case["kind"] == "normals":
        if case.get("mem") == "host":
            state["xyz"] = [v.cpu().numpy() for v in xyz]
            state["out"] = np.zeros((n, 3), np.float32)
        else:
            state["out"] = torch.zeros(n, 3, device="cuda")
        if case.get("learned"):
            g = _generator(seed + 7_919)
            held_out = _shuffled(g, _CLOUDS[case["cloud"]](g, n))
            torch.cuda.synchronize()
            ctx.build(*held_out)
            train_radius_model(ctx, k, steps=500, seed=seed % 1000, max_rows=131_072)
            ctx.set_learned(True, skip_seed=True)
    elif case["kind"] == "lists":
        state["idx"] = torch.zeros(n, k, dtype=torch.int32, device="cuda")
        state["d2"] = torch.zeros(n, k, device="cuda")
    elif case["kind"] == "queries":
        # the second scan: points near the map's own, in no useful order
        g = _generator(seed + 104_729)
        m = case["queries"]
        pick = torch.randint(n, (m,), generator=g, device="cuda")
        near = torch.stack([v[pick] for v in xyz], 1)
        state["queries"] = (near + 0.003 * torch.randn(m, 3, generator=g, device="cuda")).contiguous()
        torch.cuda.synchronize()
        ctx.build(*xyz)
    elif case["kind"] == "train":
        torch.cuda.synchronize()
        ctx.build(*xyz)
        order = np.random.default_rng(seed).permutation(ctx.info()["n_points"])
        state["features"] = np.ascontiguousarray(ctx.features()[order])
        state["targets"] = np.ascontiguousarray(radius_targets(ctx, k)[order])
    torch.cuda.synchronize()
    return state


def _batch_layout(case, seed):
    rng = np.random.default_rng(seed)
    sizes = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["clouds"])).astype(np.int64)
    offsets = np.zeros(case["clouds"] + 1, np.int64)
    offsets[1:] = np.cumsum(sizes)
    return sizes, offsets, rng.choice(np.asarray([8, 16, 32], np.int32), case["clouds"])


def _prepare_batch(case, seed):
    # one layout for all seeds (the same fleet of sensors), other points for each
    sizes, offsets, ks = _batch_layout(case, 1)
    g = _generator(seed)
    clouds = [_shuffled(g, _scene(g, int(m))) for m in sizes]
    xyz = [torch.cat([c[i] for c in clouds]) for i in range(3)]
    state = {"case": case, "ctx": Context(), "xyz": xyz, "ks": ks, "offsets": offsets,
             "out": torch.zeros(int(offsets[-1]), 3, device="cuda")}
    torch.cuda.synchronize()
    return state


# ---- one pass ----------------------------------------------------------------


# Output buffers hold one row per input point, kept by the caller; equal codes
# leave fewer tree points, and the rows past them stay as they were (zero).


def run(state):
    case, ctx = state["case"], state["ctx"]
    if case["kind"] == "batch":
        out, _, u = ctx.normals_batch(state["xyz"], (state["ks"], state["offsets"]), out=state["out"])
        return {"normals": out, "points": u}
    if case["kind"] == "queries":
        idx, d2 = ctx.knn(state["queries"], case["k"], with_d2=True)
        return {"idx": idx, "d2": d2}
    if case["kind"] == "train":
        ctx.mlp_init(1)
        losses = ctx.mlp_train(state["features"], state["targets"], case["steps"], case["batch"], 2e-3)
        return {"losses": losses, "params": ctx.mlp_params()}
    if case.get("mem") == "host":
        octree = Octree(RadixTree(PointCloud(*state["xyz"]), context=ctx))
        NormalEstimation.estimateNormals(octree, k=case["k"], out=state["out"][:octree.n_pts])
        return {"normals": state["out"], "points": octree.n_pts}
    u = ctx.build(*state["xyz"])["n_points"]
    if case["kind"] == "lists":
        ctx.knn_self(case["k"], with_d2=True, out=state["idx"][:u], out_d2=state["d2"][:u])
        return {"idx": state["idx"], "d2": state["d2"], "points": u}
    ctx.normals(case["k"], out=state["out"][:u])
    return {"normals": state["out"], "points": u}


def work(case):
    """Inputs read once, outputs written once; the arithmetic of the neighbours that end up in the lists
    (8 operations a distance, 18 a covariance term) and about 300 for an eigensolve."""
    if case["kind"] == "batch":
        sizes, _, ks = _batch_layout(case, 1)
        return {"bytes": int(24 * sizes.sum()), "flops": int((sizes * (26 * ks.astype(np.int64) + 300)).sum())}
    n, k = case["n"], case["k"]
    if case["kind"] == "train":
        rows = case["steps"] * min(case["batch"], n)
        return {"bytes": 132 * n + 4 * case["steps"] + 4 * 6_337, "flops": 6 * 6_208 * rows}
    if case["kind"] == "queries":
        return {"bytes": (12 + 8 * k) * case["queries"] + 12 * n, "flops": 8 * k * case["queries"]}
    if case["kind"] == "lists":
        return {"bytes": (12 + 8 * k) * n, "flops": 8 * k * n}
    return {"bytes": 24 * n, "flops": (26 * k + 300) * n}


# ---- the same in 64 bits ------------------------------------------------------


def _tree_points(xyz, code_bits):
    """The tree's points: Morton codes as the reference forms them (32-bit by definition), the unique ones
    in ascending order, decoded."""
    bits = code_bits // 3
    top = torch.tensor(float((1 << bits) - 1), device="cuda")
    lo = torch.stack([v.min() for v in xyz]).min()
    span = torch.stack([v.max() for v in xyz]).max() - lo
    cell = [((v - lo) / span * top).long() & ((1 << bits) - 1) for v in xyz]
    code = torch.zeros_like(cell[0])
    for b in range(bits):
        for a in range(3):
            code |= ((cell[a] >> b) & 1) << (3 * b + a)
    code = torch.unique(code)
    axes = []
    for a in range(3):
        c = torch.zeros_like(code)
        for b in range(bits):
            c |= ((code >> (3 * b + a)) & 1) << b
        axes.append(((c.float() / top).double() * span.double() + lo.double()).float())
    return torch.stack(axes, 1).double()


def _nearest(points, queries, k):
    idx, d2 = [], []
    rows = max(1, 150_000_000 // points.shape[0])
    for q in queries.split(rows):
        d = (q[:, 0:1] - points[:, 0]) ** 2
        for a in (1, 2):
            d += (q[:, a:a + 1] - points[:, a]) ** 2
        v, i = d.topk(k, dim=1, largest=False)
        idx.append(i)
        d2.append(v)
    return torch.cat(idx), torch.cat(d2)


def _rows(t, n):
    return torch.cat([t.cpu(), torch.zeros(n - t.shape[0], t.shape[1], dtype=t.dtype)])


def exact(case, seed):
    if case["kind"] in ("batch", "train") or case.get("compat") or case["n"] > EXACT_POINTS:
        return None
    if case["kind"] == "queries" and case["queries"] * case["n"] > EXACT_POINTS**2:
        return None
    state = prepare({**case, "learned": False}, seed)
    xyz = [torch.as_tensor(v, device="cuda") for v in state["xyz"]]
    points = _tree_points(xyz, case.get("code_bits", 63))
    k = case["k"]
    if case["kind"] == "queries":
        return {"idx": None, "d2": _nearest(points, state["queries"].double(), k)[1].cpu()}
    idx, d2 = _nearest(points, points, k)
    if case["kind"] == "lists":
        return {"idx": None, "d2": _rows(d2, case["n"]), "points": None}
    near = points[idx] - points.unsqueeze(1)
    near = near - near.mean(1, keepdim=True)
    cov = (near.transpose(1, 2) @ near / max(k - 1, 1)).cpu()
    normal = torch.linalg.eigh(cov)[1][:, :, 0]
    away = (normal * points.cpu()).sum(1, keepdim=True) > 0  # viewpoint at the origin
    return {"normals": _rows(torch.where(away, -normal, normal), case["n"]), "points": None}
