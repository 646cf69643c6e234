"""Performance cases of the registration engine: the calls that a program makes
through the public Python API, from a toy lookup to a large resident model.

A case is a dict of plain values.  ``listed()`` names the cases that are
tracked, ``draw(rng)`` gives further ones of the same ranges, ``prepare``
builds what a program holds before the call, ``run`` is one call and
``work`` counts what the call cannot do without.  Every cloud is synthetic
(shape families, occlusion, clutter and noise of ``synthetic.py``).
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("ppf-registration-spatial-hashing_b200")
syn = pkg.synthetic

FAMILIES = ("superellipsoid", "torus", "capsules", "spheres_slab")
# The four models of the multi-model scene and their tau_d (the benchmark's).
MULTI_TAU = (0.03, 0.035, 0.03, 0.05)


def _lookup(name, family, n_model, n_scene, tau, df, **kw):
    case = {"name": name, "kind": "lookup", "family": family, "n_model": n_model, "n_scene": n_scene,
            "tau": tau, "df": df, "thr": 0.3, "sigma": 5e-4, "tilt": 2.0, "mode": "plain"}
    case.update(kw)
    return case


def listed():
    return [
        # The smallest call: a coarse model in a small cropped scene, where
        # launches, synchronisations and allocations are most of the time.
        _lookup("lookup_tiny", "superellipsoid", 200, 700, 0.05, 5),
        # One model in one scene at the plain method's sizes.
        _lookup("lookup_plain", "superellipsoid", 2000, 10000, 0.05, 5),
        # Odd sizes, per-point vote weights and the L1 clustering option.
        _lookup("lookup_weighted_l1", "capsules", 3511, 20011, 0.04, 7, mode="weighted_l1"),
        # Averaged clusters on a flat-faced model: many kept poses, so the
        # clustering carries as much of the call as the votes.
        _lookup("lookup_averaged", "spheres_slab", 3047, 24007, 0.05, 41, mode="averaged", tilt=0.0),
        # Greedy pose clustering (the cpu_clustering option).
        _lookup("lookup_greedy", "torus", 1501, 6007, 0.05, 9, mode="greedy"),
        # A large resident model against a large scan, few reference points.
        _lookup("lookup_large", "capsules", 20000, 200003, 0.04, 4001),
        # The benchmark's multi-model scene: four models rebuilt and looked up
        # per call, at a fifth of its scene reference points.
        {"name": "register_multi", "kind": "register_multi", "n_scene": 60000, "df": 25, "thr": 0.3, "avg": False},
        # The drop-in call of a short program: host clouds, no context kept.
        {"name": "register_once", "kind": "register_once", "n_model_a": 1500, "n_model_b": 2511,
         "n_scene_a": 4000, "n_scene_b": 7013, "tau": 0.05, "df": 5, "thr": 0.4},
        # A large model registered once against a small scene: the build of
        # its hash array is the call.
        {"name": "register_build", "kind": "register_build", "family": "torus", "n_model": 14003, "n_scene": 4001,
         "tau": 0.04, "df": 101, "thr": 0.4},
        # Scenes of uneven sizes against a resident library, one batched call.
        {"name": "batch_library", "kind": "batch", "n_models": 4, "model_lo": 2000, "model_hi": 6000, "n_requests": 10,
         "scene_lo": 5000, "scene_hi": 40000, "tau": 0.04, "df": 23, "thr": 0.3},
        # The same library behind the request loop: host scenes submitted at
        # once, every result awaited.
        {"name": "served_library", "kind": "served", "n_models": 4, "model_lo": 2000, "model_hi": 6000,
         "n_requests": 12, "scene_lo": 3000, "scene_hi": 20000, "tau": 0.04, "df": 23, "thr": 0.3},
        # The driver's preparation of a raw scan and a dense model: extents,
        # d_dist and voxel-grid downsampling of host clouds.
        {"name": "preprocess_scan", "kind": "preprocess", "n_scan": 1_000_003, "n_model": 150_001, "tau": 0.05,
         "leaf": 0.006},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# Expected run length of a matched scene pair as a share of the n^2 model
# pairs, over all scene pairs, by family (sampled on the generated scenes).
_MATCH = {"superellipsoid": 1.2e-4, "torus": 2e-5, "capsules": 1.2e-5, "spheres_slab": 2e-4}


def _votes(family, n_model, n_scene, df):
    return math.ceil(n_scene / df) * n_scene * float(n_model) ** 2 * _MATCH[family]


def draw(rng):
    kind = rng.choice(["lookup", "lookup", "lookup", "lookup", "register_once", "register_build", "batch", "served",
                       "preprocess"])
    if kind == "lookup":
        family = rng.choice(FAMILIES)
        mode = rng.choice(["plain", "plain", "plain", "weighted_l1", "averaged", "greedy"])
        n_model = _log_int(rng, 150, 12000 if mode == "plain" else 3000)
        n_scene = _log_int(rng, max(500, n_model), 120000 if mode == "plain" else 20000)
        df = rng.choice([3, 5, 5, 7, 10, 25])
        limit = 8e10 if mode == "plain" else 4e9
        while _votes(family, n_model, n_scene, df) > limit:
            df = df * 2 + 1
        if mode in ("averaged", "greedy"):
            df = max(df, 9)
        case = _lookup("", family, n_model, n_scene, rng.choice([0.04, 0.05]), df, mode=mode,
                       thr=rng.choice([0.3, 0.4]) if mode != "greedy" else 0.5, tilt=rng.choice([0.0, 2.0]))
        del case["name"]
        return case
    if kind == "register_once":
        return {"kind": kind, "n_model_a": _log_int(rng, 200, 2500), "n_model_b": _log_int(rng, 200, 2500),
                "n_scene_a": _log_int(rng, 2600, 9000), "n_scene_b": _log_int(rng, 2600, 9000),
                "tau": rng.choice([0.04, 0.05]), "df": rng.choice([5, 10]), "thr": 0.4}
    if kind == "register_build":
        return {"kind": kind, "family": rng.choice(["torus", "capsules"]), "n_model": _log_int(rng, 2000, 14000),
                "n_scene": _log_int(rng, 1000, 6000), "tau": rng.choice([0.03, 0.04]), "df": 101, "thr": 0.4}
    if kind in ("batch", "served"):
        return {"kind": kind, "n_models": rng.randint(2, 5), "model_lo": 1000, "model_hi": _log_int(rng, 1500, 5000),
                "n_requests": rng.randint(3, 12), "scene_lo": 2000, "scene_hi": _log_int(rng, 4000, 20000),
                "tau": rng.choice([0.04, 0.05]), "df": rng.choice([23, 31]), "thr": rng.choice([0.3, 0.4])}
    return {"kind": kind, "n_scan": _log_int(rng, 20000, 1_000_000), "n_model": _log_int(rng, 5000, 150000),
            "tau": rng.choice([0.03, 0.05]), "leaf": rng.choice([0.004, 0.006, 0.01])}


# ------------------------------------------------------------------ inputs


def _scene(rng, models, n_scene, sigma=5e-4, tilt=0.0, occlusion=0.3):
    """The models under random poses, each occluded, on a ground plane with
    three boxes: exactly n_scene points when the clutter has room for it."""
    parts = []
    for k, m in enumerate(models):
        t = np.array([0.32 * (k % 2), 0.32 * (k // 2), 0.0]) + rng.uniform(-0.03, 0.03, 3)
        pose = np.eye(4)
        pose[:3, :3] = syn.uniform_rotation(rng)
        pose[:3, 3] = t
        inst = syn.occlude(rng, syn.transform(m, pose), occlusion)
        if len(inst) > max(n_scene // (2 * len(models)), 1):  # a sparser scan than the model
            inst = inst.subset(rng.choice(len(inst), max(n_scene // (2 * len(models)), 1), replace=False))
        parts.append(inst)
    clutter = n_scene - sum(len(p) for p in parts)
    n_plane = int(0.6 * clutter)
    half = 0.3 + 0.16 * min(len(models), 2)
    parts.append(syn.ground_plane(rng, n_plane, -0.16, half, (0.16, 0.16) if len(models) > 1 else (0.0, 0.0)))
    per = rng.multinomial(clutter - n_plane, np.ones(3) / 3)
    for b in range(3):
        side = rng.uniform(0.05, 0.12, size=3)
        at = rng.uniform(-half + 0.08, half - 0.08, size=2)
        lo = np.array([at[0], at[1], -0.16])
        parts.append(syn.box_surface(rng, per[b], lo, lo + side, faces=5))
    return syn.add_noise(rng, syn.Cloud.concat(parts), sigma, tilt)


def _dev(cloud):
    return (torch.from_numpy(np.ascontiguousarray(cloud.points)).cuda(),
            torch.from_numpy(np.ascontiguousarray(cloud.normals)).cuda())


def _host(cloud):
    return np.ascontiguousarray(cloud.points), np.ascontiguousarray(cloud.normals)


def _sizes(case):
    """Model and request sizes of a library case (from its own numbers, not from the seed)."""
    n, r = case["n_models"], case["n_requests"]
    at = lambda lo, hi, k, m: int(lo * (hi / lo) ** (k / max(m - 1, 1)))  # noqa: E731
    models = [at(case["model_lo"], case["model_hi"], k, n) for k in range(n)]
    scenes = [at(case["scene_lo"], case["scene_hi"], (k * 7) % r, r) for k in range(r)]
    return models, scenes


def prepare(case, seed):
    rng = np.random.default_rng([seed, 7])
    kind = case["kind"]
    if kind == "lookup":
        ctx = pkg.Context(0)
        cloud = syn.make_shape(rng, case["family"], case["n_model"])
        d = syn.d_dist_for(cloud, case["tau"])
        mode = case["mode"]
        model = pkg.Model(_dev(cloud), d, case["thr"], cpu_clustering=mode == "greedy",
                          use_l1_norm=mode == "weighted_l1", use_averaged_clusters=mode == "averaged", context=ctx)
        if mode == "weighted_l1":
            model.SetModelPointVoteWeights(rng.uniform(0.5, 2.0, case["n_model"]).astype(np.float32))
        scene = _scene(rng, [cloud], case["n_scene"], case["sigma"], case["tilt"])
        return {"case": case, "ctx": ctx, "model": model, "scene": _dev(scene), "d": d}
    if kind == "register_multi":
        spec = syn.config_multi_model(seed=1001 + seed, n_scene=case["n_scene"], tau_d=MULTI_TAU,
                                      sizes=[5711, 4838, 5461, 3047])
        return {"case": case, "ctx": pkg.Context(0), "models": [_dev(m) for m in spec.models],
                "scene": _dev(spec.scene), "d": list(spec.d_dists)}
    if kind == "register_once":
        models = [syn.make_shape(rng, "superellipsoid", case["n_model_a"]),
                  syn.make_shape(rng, "capsules", case["n_model_b"])]
        scenes = [_scene(rng, models, n, 5e-4, 2.0) for n in (case["n_scene_a"], case["n_scene_b"])]
        return {"case": case, "models": [_host(m) for m in models], "scenes": [_host(s) for s in scenes],
                "d": [syn.d_dist_for(m, case["tau"]) for m in models]}
    if kind == "register_build":
        cloud = syn.make_shape(rng, case["family"], case["n_model"])
        return {"case": case, "ctx": pkg.Context(0), "models": [_dev(cloud)],
                "scene": _dev(_scene(rng, [cloud], case["n_scene"], 5e-4, 2.0)),
                "d": [syn.d_dist_for(cloud, case["tau"])]}
    if kind in ("batch", "served"):
        ctx = pkg.Context(0)
        sizes, scene_sizes = _sizes(case)
        clouds = [syn.make_shape(rng, FAMILIES[k % 4], n) for k, n in enumerate(sizes)]
        d = [syn.d_dist_for(c, case["tau"]) for c in clouds]
        models = [pkg.Model(_dev(c), x, case["thr"], context=ctx) for c, x in zip(clouds, d)]
        ids = [(k * 3 + 1) % len(clouds) for k in range(len(scene_sizes))]
        scenes = [_scene(rng, [clouds[i], clouds[(i + 1) % len(clouds)]], n) for i, n in zip(ids, scene_sizes)]
        state = {"case": case, "ctx": ctx, "models": models, "d": d, "ids": ids}
        if kind == "batch":
            state["scenes"] = [_dev(s) for s in scenes]
        else:
            ctx.synchronize()
            state["scenes"] = [_host(s) for s in scenes]
            state["server"] = pkg.Server(models, memory_budget=24 << 30, workers=1, max_batch=8)
        return state
    scan = [syn.make_shape(rng, FAMILIES[k], 40000) for k in range(4)]
    per = case["n_scan"]
    scene = _scene(rng, scan, per, 1e-3, 2.0, 0.4)
    model = syn.make_shape(rng, "capsules", case["n_model"])
    cs, cm = _voxel_capacity(case)
    return {"case": case, "ctx": pkg.Context(0), "scenes": [_host(scene)], "models": [_host(model)],
            "out": [np.zeros((k, 3), np.float32) for k in (cs, cs, cm, cm)]}


def _voxel_capacity(case):
    """Voxels a preprocessed scan and model can fill: surfaces of at most 2
    square metres and 0.05, at up to three noisy layers of voxels."""
    return (min(case["n_scan"], int(6.0 / case["leaf"] ** 2)),
            min(case["n_model"], int(0.15 / (case["tau"] * 0.05) ** 2)))


# -------------------------------------------------------------------- pass


def _counts(stats):
    return np.array([stats["n_votes"], stats["n_matched_pairs"], stats["max_vote_count"], stats["n_kept"],
                     stats["max_idx"]], np.int64)


def _into(out, points):
    """Voxel means into the program's own array (their number depends on the cloud)."""
    out[: len(points)] = points
    out[len(points):] = 0.0
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "lookup":
        model = state["model"]
        scene = pkg.Scene(state["scene"], state["d"], case["df"], context=state["ctx"])
        pose = model.ppf_lookup(scene)
        return {"pose": pose, "counts": _counts(model.stats), "score": np.float32(model.stats["best_score"])}
    if kind in ("register_multi", "register_build"):
        poses, stats = pkg.ppf_registration([state["scene"]], state["models"], state["d"], case["df"], case["thr"],
                                            use_averaged_clusters=case.get("avg", False), context=state["ctx"],
                                            return_stats=True)
        return {"poses": np.array(poses), "counts": np.array([[_counts(s) for s in row] for row in stats])}
    if kind == "register_once":
        return {"poses": np.array(pkg.ppf_registration(state["scenes"], state["models"], state["d"], case["df"],
                                                       case["thr"]))}
    if kind == "batch":
        models = [state["models"][i] for i in state["ids"]]
        scenes = [pkg.Scene(s, state["d"][i], case["df"], context=state["ctx"])
                  for s, i in zip(state["scenes"], state["ids"])]
        poses, stats = pkg.lookup_batch(models, scenes, context=state["ctx"], return_stats=True)
        return {"poses": poses, "counts": np.array([_counts(s) for s in stats])}
    if kind == "served":
        server = state["server"]
        tickets = [server.submit(s, [i], case["df"]) for s, i in zip(state["scenes"], state["ids"])]
        got = [server.wait(t) for t in tickets]
        return {"poses": np.array([g[0][0] for g in got]), "counts": np.array([_counts(g[1][0]) for g in got])}
    scenes, models, d = pkg.preprocess(state["scenes"], state["models"], [case["tau"]], case["leaf"],
                                       context=state["ctx"])
    sp, sn, mp, mn = state["out"]
    return {"scene_points": _into(sp, scenes[0][0]), "scene_normals": _into(sn, scenes[0][1]),
            "model_points": _into(mp, models[0][0]), "model_normals": _into(mn, models[0][1]),
            "d_dist": np.array(d, np.float32)}


def work(case):
    """Clouds and hash arrays read once, poses and kept votes written once;
    operations: 40 per scene pair evaluated (feature, quantisation, key), 12
    per model pair keyed and sorted, 4 per vote (angle, bin, cell, count).
    The votes are the expectation of the case's sizes and shape family."""
    kind = case["kind"]
    cloud = 24

    def lookup(family, n, s, df):
        pairs = math.ceil(s / df) * s
        return 40 * pairs + 4 * _votes(family, n, s, df)

    if kind == "lookup":
        n, s = case["n_model"], case["n_scene"]
        return {"bytes": cloud * s + 4 * n * n + 64, "flops": lookup(case["family"], n, s, case["df"])}
    if kind == "register_multi":
        sizes, s = [5711, 4838, 5461, 3047], case["n_scene"]
        return {"bytes": cloud * (s + sum(sizes)) + sum(20 * n * n for n in sizes) + 256,
                "flops": sum(52 * n * n + lookup(f, n, s, case["df"]) for f, n in zip(FAMILIES, sizes))}
    if kind == "register_build":
        n, s = case["n_model"], case["n_scene"]
        return {"bytes": cloud * (s + n) + 20 * n * n + 64,
                "flops": 52 * n * n + lookup(case["family"], n, s, case["df"])}
    if kind == "register_once":
        ms, ss = (case["n_model_a"], case["n_model_b"]), (case["n_scene_a"], case["n_scene_b"])
        return {"bytes": cloud * (sum(ms) + sum(ss)) + sum(20 * n * n for n in ms) + 256,
                "flops": sum(52 * n * n for n in ms) + sum(lookup(f, n, s, case["df"]) for s in ss
                                                           for f, n in zip(("superellipsoid", "capsules"), ms))}
    if kind in ("batch", "served"):
        sizes, scenes = _sizes(case)
        ids = [(k * 3 + 1) % len(sizes) for k in range(len(scenes))]
        return {"bytes": sum(cloud * s + 64 for s in scenes) + sum(4 * sizes[i] ** 2 for i in set(ids)),
                "flops": sum(lookup(FAMILIES[i % 4], sizes[i], s, case["df"]) for i, s in zip(ids, scenes))}
    n = case["n_scan"] + case["n_model"]
    return {"bytes": 2 * cloud * n, "flops": 40 * n}


# ------------------------------------------------------------------- exact


def _voxel_mean(points, normals, leaf):
    """Voxel means in 64 bits; the voxel of a point is the float32 rule itself."""
    inv = np.float32(1.0) / np.float32(leaf)
    low = np.floor(points.min(0) * inv).astype(np.int64)
    high = np.floor(points.max(0) * inv).astype(np.int64)
    dim = high - low + 1
    cell = (np.floor(points * inv) - low.astype(np.float32)).astype(np.int64)
    index = cell[:, 0] + cell[:, 1] * dim[0] + cell[:, 2] * dim[0] * dim[1]
    _, inverse, count = np.unique(index, return_inverse=True, return_counts=True)
    mean = lambda v: np.stack([np.bincount(inverse, v[:, k].astype(np.float64)) for k in range(3)], 1) / count[:, None]  # noqa: E731
    return mean(points), mean(normals)


def exact(case, seed):
    if case["kind"] != "preprocess":
        # A pose is one kept vote's transform, picked among votes that exist
        # only through 32-bit quantisation: 64 bits give other votes.
        return None
    rng = np.random.default_rng([seed, 7])
    scan = [syn.make_shape(rng, FAMILIES[k], 40000) for k in range(4)]
    scene = _scene(rng, scan, case["n_scan"], 1e-3, 2.0, 0.4)
    model = syn.make_shape(rng, "capsules", case["n_model"])
    d = float(np.float32(case["tau"]) * np.max(model.points.max(0) - model.points.min(0)))
    sp, sn = _voxel_mean(scene.points, scene.normals, case["leaf"])
    mp, mn = _voxel_mean(model.points, model.normals, d)
    ext = model.points.max(0).astype(np.float64) - model.points.min(0).astype(np.float64)
    cs, cm = _voxel_capacity(case)

    def padded(v, capacity):
        return np.concatenate([v, np.zeros((capacity - len(v), 3))])

    return {"scene_points": padded(sp, cs), "scene_normals": padded(sn, cs), "model_points": padded(mp, cm),
            "model_normals": padded(mn, cm), "d_dist": np.array([float(np.float32(case["tau"])) * ext.max()])}
