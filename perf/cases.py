"""The work a renderer has this library do, as measurable cases.

Each case names a path (`kind`), its sizes and its options.  `prepare` makes what a program holds
before the call (scene, tracer, guide, input arrays, all on the GPU, from the seed alone), `run`
is one pass through the public entry points, `work` the bytes and operations the pass cannot do
without, and `exact` the same result in 64-bit arithmetic where the result is a computed number
(not a Monte Carlo estimate whose value depends on single-precision path decisions).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from rtlib_b200 import scenes
from rtlib_b200.hashgrid import KEY_MORTON, KEY_REFERENCE, HashGrid, MortonQuadTreeController, MortonQuadTrees
from rtlib_b200.mlp import MLPGuide
from rtlib_b200.sdtree import SDTree, SDTreeController
from rtlib_b200.tracer import FLAG_BUILD, FLAG_NEE, FLAG_RIS, Scene, Tracer

DEV = "cuda"
ROOMS_AABB = ((-0.005,) * 3, (14.005, 4.005, 10.005))
BOX_AABB = ((-0.005,) * 3, (1.005,) * 3)
FLAGS = {"DEF": 0, "NEE": FLAG_NEE, "RIS": FLAG_NEE | FLAG_RIS}


def listed():
    return [
        # the first image of an interactive viewport after a camera move: one sample of a small
        # image; launches and their gaps are most of it
        {"name": "viewport_96x54", "kind": "render", "width": 96, "height": 54, "depth": 8, "spp": 1, "tracer": "NEE",
         "materials": "lambert"},
        # SD-tree guided path tracing of the Cornell box under the pass controller (record, build,
        # refine, guided sampling): a draft-quality budget at the usual image size
        {"name": "cornell_sdtree_512", "kind": "guided", "width": 512, "height": 512, "depth": 8, "budget": 63,
         "tracer": "NEE"},
        # hash-grid guided path tracing of the million-triangle occluded scene, RIS with 32
        # candidates: the large offline render
        {"name": "occluded_hashgrid_1280x720", "kind": "grid", "width": 1280, "height": 720, "depth": 16, "budget": 7,
         "objects": 2048, "lights": 4096, "level": 3, "candidates": 32},
        # one recording pass of the learned guide on the same scene: network inference between
        # the bounces, trace vertices kept as training records
        {"name": "occluded_learned_640x360", "kind": "learned", "width": 640, "height": 360, "depth": 16, "spp": 2,
         "objects": 2048, "lights": 4096, "level": 3, "candidates": 32},
        # differentiable rendering: one optimisation step's primal image and its gradients
        # towards an albedo texture and the emitters of the split ceiling light
        {"name": "cornell_adjoint_256", "kind": "adjoint", "width": 256, "height": 256, "depth": 8, "spp": 16,
         "texture": 256, "light_grid": 4},
        # the SD-tree by itself, driven by another renderer: a cleared tree learns 2^20 records
        # over two passes, then answers 2^22 sample + pdf queries
        {"name": "sdtree_pass_1m", "kind": "sdtree", "records": 1 << 20, "queries": 1 << 22, "passes": 2,
         "canonical": True},
        # a kept SD-tree queried for a small batch of shading points (a tile of another renderer)
        {"name": "sdtree_query_3001", "kind": "sdtree_query", "queries": 3001, "records": 1 << 18, "passes": 3},
        # the hash grid's cells located for a pass: insert of a surface sampling, lookup of a
        # frame's shading points
        {"name": "hashgrid_512k", "kind": "hashgrid", "points": 1 << 19, "queries": 1 << 22, "slots": 1 << 20,
         "morton": True},
        # the grid's Morton quadtrees: a frame's records, the rebuild of every sampling pyramid, a
        # frame's sample + pdf queries
        {"name": "morton_trees_1m", "kind": "trees", "cells": 1 << 20, "level": 4, "queries": 1 << 22, "used": 0.36},
        # the learned guide trained on the records of one pass
        {"name": "mlp_train_256k", "kind": "mlp_train", "records": 1 << 18, "batch": 1 << 14, "epochs": 1},
        # the learned guide's mixture for a frame of shading points
        {"name": "mlp_eval_1m", "kind": "mlp_eval", "samples": 1 << 20, "raw": False},
        # closest hits and visibility of a frame's rays in the million-triangle scene (the
        # hit-query boundary used by itself)
        {"name": "hits_1m", "kind": "hits", "rays": 1 << 20, "objects": 2048, "lights": 4096, "level": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "guided", "grid", "learned", "adjoint", "sdtree", "sdtree_query", "hashgrid", "trees",
                       "mlp_train", "mlp_eval", "hits"])
    if kind == "render":
        return {"kind": kind, "width": _log_int(rng, 16, 800), "height": _log_int(rng, 16, 600),
                "depth": rng.randint(2, 12), "spp": _log_int(rng, 1, 16), "tracer": rng.choice(["DEF", "NEE", "RIS"]),
                "materials": rng.choice(["lambert", "lambert", "glass_phong"])}
    if kind == "guided":
        return {"kind": kind, "width": _log_int(rng, 64, 700), "height": _log_int(rng, 64, 520),
                "depth": rng.randint(4, 12), "budget": _log_int(rng, 7, 100), "tracer": rng.choice(["DEF", "NEE", "RIS"])}
    rooms = {"objects": _log_int(rng, 64, 800), "lights": 2 * _log_int(rng, 32, 1024), "level": rng.randint(1, 3)}
    if kind == "grid":
        return {"kind": kind, "width": _log_int(rng, 160, 900), "height": _log_int(rng, 90, 500),
                "depth": rng.randint(4, 16), "budget": rng.choice([3, 7]), **rooms, "candidates": rng.choice([8, 16, 32])}
    if kind == "learned":
        return {"kind": kind, "width": _log_int(rng, 96, 640), "height": _log_int(rng, 54, 360),
                "depth": rng.randint(4, 16), "spp": rng.randint(1, 3), **rooms, "candidates": rng.choice([8, 16, 32])}
    if kind == "adjoint":
        return {"kind": kind, "width": _log_int(rng, 40, 400), "height": _log_int(rng, 40, 400),
                "depth": rng.randint(3, 10), "spp": _log_int(rng, 2, 24), "texture": _log_int(rng, 16, 300),
                "light_grid": rng.randint(1, 4)}
    if kind == "sdtree":
        return {"kind": kind, "records": _log_int(rng, 1 << 13, 1 << 21), "queries": _log_int(rng, 1 << 12, 1 << 23),
                "passes": rng.randint(1, 4), "canonical": rng.choice([True, False])}
    if kind == "sdtree_query":
        return {"kind": kind, "queries": _log_int(rng, 33, 1 << 21), "records": _log_int(rng, 1 << 14, 1 << 20),
                "passes": rng.randint(1, 4)}
    if kind == "hashgrid":
        points = _log_int(rng, 500, 1 << 21)
        return {"kind": kind, "points": points, "queries": _log_int(rng, 1 << 12, 1 << 22),
                "slots": 1 << rng.randint(max(10, points.bit_length() - 1), 22), "morton": rng.choice([True, False])}
    if kind == "trees":
        level = rng.randint(2, 6)
        return {"kind": kind, "cells": _log_int(rng, 100, min(1 << 20, (1 << 28) >> (2 * level))), "level": level,
                "queries": _log_int(rng, 1 << 12, 1 << 22), "used": rng.choice([0.1, 0.36, 0.8, 1.0])}
    if kind == "mlp_train":
        return {"kind": kind, "records": _log_int(rng, 3000, 1 << 18), "batch": _log_int(rng, 1 << 10, 1 << 15),
                "epochs": rng.randint(1, 2)}
    if kind == "mlp_eval":
        return {"kind": kind, "samples": _log_int(rng, 100, 1 << 21), "raw": rng.choice([True, False])}
    return {"kind": kind, "rays": _log_int(rng, 1 << 12, 1 << 21), **rooms}


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=4)
def _rooms(objects, lights, level):
    # the scene file of the occluded rooms: the same geometry for every seed
    return scenes.occluded_rooms(16, 9, n_objects=objects, n_lights=lights, sphere_level=level)


def _rooms_of(case, width, height):
    sc = dict(_rooms(case["objects"], case["lights"], case["level"]))
    # the camera scenes.occluded_rooms sets up for this image's aspect ratio
    sc["camera"] = scenes._camera((7.5, 1.6, 3.6), (10.0, 1.0, 5.0), (0, 1, 0), 60.0, width / height)
    sc["width"], sc["height"] = width, height
    return sc


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _unit(n, g):
    v = torch.randn((n, 3), generator=g, device=DEV)
    return (v / v.norm(dim=1, keepdim=True)).contiguous()


def _vmf4(n, g, kappa=50.0):
    """Directions of a 4-lobe von Mises-Fisher mixture: radiance that arrives from few sides."""
    axes = _unit(4, g)
    mu = axes[torch.randint(0, 4, (n,), generator=g, device=DEV)]
    u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    w = (1.0 + torch.log(u + (1.0 - u) * math.exp(-2.0 * kappa)) / kappa).float()
    t = torch.linalg.cross(mu, _unit(n, g))
    t = t / t.norm(dim=1, keepdim=True)
    d = w[:, None] * mu + torch.sqrt((1.0 - w * w).clamp_min(0.0))[:, None] * t
    return (d / d.norm(dim=1, keepdim=True)).contiguous()


def _canonical(d):
    phi = torch.atan2(d[:, 1], d[:, 0])
    phi = torch.where(phi < 0, phi + 2.0 * math.pi, phi)
    return torch.stack([(d[:, 2].clamp(-1, 1) + 1.0) / 2.0, (phi / (2.0 * math.pi)).clamp(0.0, 1.0)], 1).contiguous()


def _seeds(n, g):
    return torch.randint(1, 2**31 - 1, (n,), generator=g, device=DEV, dtype=torch.int32)


def _lognormal(n, g):
    return torch.exp(torch.randn(n, generator=g, device=DEV))


def _threshold(case, it):
    # the standalone workload's 12000 sqrt(2^iter) at 2^20 records, in proportion to the records
    return int(12000.0 * math.sqrt(2.0 ** it) * case["records"] / (1 << 20)) + 1


def _surface(tri, n, g):
    """n points uniform by area on the triangles tri (nt, 9)."""
    v = tri.view(-1, 3, 3)
    c = torch.cumsum(torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]).double().norm(dim=1), 0)
    k = torch.searchsorted(c, torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * c[-1]).clamp_max(len(v) - 1)
    ab = torch.rand((n, 2), generator=g, device=DEV)
    ab = torch.where(ab.sum(1, keepdim=True) > 1.0, 1.0 - ab, ab)
    t = v[k]
    return (t[:, 0] + ab[:, :1] * (t[:, 1] - t[:, 0]) + ab[:, 1:] * (t[:, 2] - t[:, 0])).contiguous()


def _weights(seed):
    """Network parameters (80 x 64, 64 x 64, 64 x 64, 64 x 48): uniform at the He bound, the last
    input and the last 8 outputs are padding."""
    g = np.random.default_rng(seed)
    out = []
    for l, (a, b) in enumerate(((80, 64), (64, 64), (64, 64), (64, 48))):
        s = math.sqrt(6.0 / (79 if l == 0 else a)) * (0.5 if l == 3 else 1.0)
        w = g.uniform(-s, s, (a, b))
        if l == 0:
            w[79] = 0.0
        if l == 3:
            w[:, 40:] = 0.0
        out.append(w.astype(np.float32).ravel())
    return np.concatenate(out)


def _shading_points(n, g):
    """Positions in the 10 m room, normals and outgoing directions."""
    return 10.0 * torch.rand((n, 3), generator=g, device=DEV), _unit(n, g), _unit(n, g)


def _rays(case, seed, tri):
    """Half camera-like rays from one eye, half bounce rays between surface points."""
    n, g = case["rays"], _gen(seed)
    h = n // 2
    eye = torch.tensor([7.5, 1.6, 3.6], device=DEV).expand(h, 3)
    cam = torch.tensor([0.6, -0.15, 0.5], device=DEV) + 0.7 * (torch.rand((h, 3), generator=g, device=DEV) - 0.5)
    p = _surface(tri, n - h, g)
    d = torch.cat([cam / cam.norm(dim=1, keepdim=True), _unit(n - h, g)])
    return torch.cat([eye, p]).contiguous(), d.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("render", "guided"):
        w, h = case["width"], case["height"]
        sc = scenes.cornell_box(w, h, materials=case.get("materials", "lambert"))
        s["tracer"] = Tracer(sc, DEV, max_depth=case["depth"], seed=seed % 1000003 + 1)
        if kind == "guided":
            s["tree"] = SDTree(*BOX_AABB, fraction=0.5)
            s["ctrl"] = SDTreeController(s["tree"], case["budget"], iteration_for_built=0, ratio_for_budget=0.5)
    elif kind in ("grid", "learned"):
        sc = _rooms_of(case, case["width"], case["height"])
        s["tracer"] = Tracer(sc, DEV, max_depth=case["depth"], num_candidates=case["candidates"], seed=seed % 1000003 + 1)
        if kind == "grid":
            s["grid"] = HashGrid(*ROOMS_AABB, (256, 64, 192), 1 << 20, keying=KEY_MORTON)
            s["trees"] = MortonQuadTrees(1 << 20, level=4, fraction=0.3)
            s["ctrl"] = MortonQuadTreeController(s["trees"], case["budget"], iteration_for_built=1, ratio_for_budget=0.5)
        else:
            s["mlp"] = MLPGuide(*ROOMS_AABB, record_capacity=1 << 18)
            s["mlp"].set_params(_weights(seed))
    elif kind == "adjoint":
        w, h, g = case["width"], case["height"], _gen(seed)
        sc = scenes.cornell_box(w, h, light_grid=case["light_grid"], back_texture=True)
        s["texture"] = 0.2 + 0.7 * torch.rand((case["texture"], case["texture"], 3), generator=g, device=DEV)
        s["tracer"] = Tracer(sc, DEV, max_depth=case["depth"], seed=seed % 1000003 + 1, textures={0: s["texture"]})
        s["target"] = 0.5 * torch.rand((h, w, 3), generator=g, device=DEV)
        s["lights"] = case["light_grid"] ** 2
    elif kind in ("sdtree", "sdtree_query"):
        n, q, g = case["records"], case["queries"], _gen(seed)
        d = _vmf4(n, g)
        s["pos"], s["radiance"] = torch.rand((n, 3), generator=g, device=DEV), _lognormal(n, g)
        s["dir"] = _canonical(d) if case.get("canonical", True) else d
        s["qpos"], s["seeds"], s["qdir"] = torch.rand((q, 3), generator=g, device=DEV), _seeds(q, g), _unit(q, g)
        s["tree"] = SDTree((0, 0, 0), (1, 1, 1))
        if kind == "sdtree_query":
            _learn(s)
    elif kind == "hashgrid":
        g = _gen(seed)
        tri = torch.from_numpy(np.ascontiguousarray(_rooms(256, 256, 2)["tri_v"])).to(DEV)
        s["points"], s["queries"] = _surface(tri, case["points"], g), _surface(tri, case["queries"], g)
        s["grid"] = HashGrid(*ROOMS_AABB, (256, 64, 192), case["slots"],
                             keying=KEY_MORTON if case["morton"] else KEY_REFERENCE)
    elif kind == "trees":
        n, g = case["queries"], _gen(seed)
        used = torch.randperm(case["cells"], generator=g, device=DEV)[: max(1, int(case["used"] * case["cells"]))]
        # some cells are seen far more often than others, and 1 % of the points have no cell
        k = (torch.rand(n, generator=g, device=DEV) ** 2 * len(used)).long().clamp_max(len(used) - 1)
        cell = used[k].int()
        s["cell"] = torch.where(torch.rand(n, generator=g, device=DEV) < 0.01, torch.full_like(cell, -1), cell)
        s["dir"], s["value"], s["seeds"] = _canonical(_vmf4(n, g)), _lognormal(n, g), _seeds(n, g)
        s["trees"] = MortonQuadTrees(case["cells"], level=case["level"])
    elif kind in ("mlp_train", "mlp_eval"):
        g = _gen(seed)
        s["mlp"] = MLPGuide((0, 0, 0), (10, 10, 10), record_capacity=1)
        s["params"] = _weights(seed)
        s["mlp"].set_params(s["params"])
        n = case.get("records") or case["samples"]
        s["points"] = _shading_points(n, g)
        if kind == "mlp_train":
            s["points"] += (_vmf4(n, g), _lognormal(n, g))
    else:
        tri = torch.from_numpy(np.ascontiguousarray(_rooms(case["objects"], case["lights"], case["level"])["tri_v"])).to(DEV)
        s["org"], s["dir"] = _rays(case, seed, tri)
        s["far"] = torch.full((case["rays"],), 2.0, device=DEV)
        s["scene"] = Scene(tri)
    return s


# ------------------------------------------------------------------ one pass
def _learn(s):
    case, tree = s["case"], s["tree"]
    tree.clear()
    for it in range(1, case["passes"] + 1):
        tree.record(s["pos"], s["dir"], s["radiance"])
        tree.build()
        tree.refine(_threshold(case, it))


def run(state):
    s = state
    case, kind = s["case"], s["case"]["kind"]
    if kind == "render":
        s["tracer"].clear()
        s["tracer"].render(case["spp"], FLAGS[case["tracer"]])
        return s["tracer"].image()
    if kind == "guided":
        s["tracer"].clear()
        s["ctrl"].start()
        s["tracer"].render_guided(s["tree"], s["ctrl"], FLAGS[case["tracer"]])
        return s["tracer"].image()
    if kind == "grid":
        s["tracer"].clear()
        s["grid"].clear()
        s["ctrl"].start()
        s["tracer"].render_grid_guided(s["grid"], s["trees"], s["ctrl"], FLAG_NEE | FLAG_RIS)
        return s["tracer"].image()
    if kind == "learned":
        s["tracer"].clear()
        s["mlp"].records(clear=True)
        s["tracer"].render_mlp(case["spp"], FLAG_NEE | FLAG_RIS | FLAG_BUILD, s["mlp"], 0.5, record_keep=0.1)
        return {"image": s["tracer"].image(), "records": s["mlp"].records()}
    if kind == "adjoint":
        tr, n = s["tracer"], 3.0 * case["width"] * case["height"]
        tr.clear()
        tr.render(case["spp"], FLAG_NEE)
        image = tr.image()
        g_tex, g_light = torch.zeros_like(s["texture"]), torch.zeros((s["lights"], 3), device=DEV)
        tr.clear()
        tr.render_adjoint(case["spp"], (2.0 / n) * (image - s["target"]), FLAG_NEE, 0, g_tex, g_light)
        return {"image": image, "texture": g_tex, "lights": g_light}
    if kind == "sdtree":
        _learn(s)
        n = case["queries"]
        d, p = torch.empty((n, 3), device=DEV), torch.empty(n, device=DEV)
        s["tree"].sample_pdf(s["qpos"], s["seeds"], out_dir=d, out_pdf_uv=p)
        return {"dir": d, "pdf": p}
    if kind == "sdtree_query":
        n = case["queries"]
        d, p, b = torch.empty((n, 3), device=DEV), torch.empty(n, device=DEV), torch.empty(n, device=DEV)
        s["tree"].sample_pdf(s["qpos"], s["seeds"], out_dir=d, out_pdf_dir=p)
        s["tree"].pdf(s["qpos"], s["qdir"], b)  # the guide's density of the renderer's own BSDF sample
        return {"dir": d, "pdf": p, "bsdf_pdf": b}
    if kind == "hashgrid":
        a = torch.empty(case["points"], dtype=torch.int32, device=DEV)
        b = torch.empty(case["queries"], dtype=torch.int32, device=DEV)
        s["grid"].clear()
        s["grid"].insert(s["points"], a)
        s["grid"].swap()
        s["grid"].lookup(s["queries"], b)
        return {"inserted": a, "found": b}
    if kind == "trees":
        n = case["queries"]
        d, p = torch.empty((n, 3), device=DEV), torch.empty(n, device=DEV)
        s["trees"].record(s["cell"], s["dir"], s["value"])
        s["trees"].update()
        s["trees"].sample_pdf(s["cell"], s["seeds"], out_dir=d, out_pdf=p)
        return {"dir": d, "pdf": p}
    if kind == "mlp_train":
        s["mlp"].set_params(s["params"])
        loss = s["mlp"].train(s["points"], batch=case["batch"], epochs=case["epochs"])
        return {"params": s["mlp"].params(), "loss": loss}
    if kind == "mlp_eval":
        return s["mlp"].eval(*s["points"], raw=case["raw"])
    n = case["rays"]
    t, uv = torch.empty(n, device=DEV), torch.empty((n, 2), device=DEV)
    prim, occ = (torch.empty(n, dtype=torch.int32, device=DEV) for _ in range(2))
    s["scene"].intersect(s["org"], s["dir"], out_t=t, out_prim=prim, out_uv=uv)
    s["scene"].intersect(s["org"], s["dir"], tmax=s["far"], any_hit=True, out_prim=occ)
    # an any-hit query tells whether something is hit, not which of several triangles
    return {"t": t, "prim": prim, "uv": uv, "occluded": occ != -1}


# ------------------------------------------------------------------ what a pass cannot do without
def _paths(case):
    """Path-bounces: about two thirds of the bounces of a depth-limited path in a closed room."""
    spp = case.get("spp") or case["budget"] + 1
    return case["width"] * case["height"] * spp, case["width"] * case["height"] * spp * max(1.0, 0.67 * case["depth"])


def _ray_flops(tris):
    # a hierarchy walk: two box tests (24 operations) a level, a few triangle tests (40)
    return 24.0 * math.log2(max(2, tris)) + 120.0


def work(case):
    kind = case["kind"]
    if kind in ("render", "guided", "adjoint"):
        paths, bounces = _paths(case)
        px = case["width"] * case["height"]
        ris = 32 if case.get("tracer") == "RIS" else 1
        rays = 1 if case.get("tracer") == "DEF" else 2
        f = bounces * (rays * _ray_flops(36) + 60.0 + (60.0 * ris if rays == 2 else 0.0))
        # the image (and, differentiated, its gradient and the texture's)
        b = 12.0 * px * (2 if kind == "adjoint" else 1) + (24.0 * case["texture"] ** 2 if kind == "adjoint" else 0)
        # a gradient pass replays the path
        return {"bytes": b, "flops": f * (2 if kind == "adjoint" else 1)}
    if kind in ("grid", "learned"):
        paths, bounces = _paths(case)
        tris = case["objects"] * 20 * 4 ** case["level"]
        f = bounces * (2 * _ray_flops(tris) + 60.0 + 60.0 * case["candidates"])
        if kind == "learned":
            f += bounces * 2.0 * (79 * 64 + 2 * 64 * 64 + 64 * 40)
        return {"bytes": 12.0 * case["width"] * case["height"] + 112.0 * tris, "flops": f}
    if kind == "sdtree":
        per = 24 if case["canonical"] else 28
        return {"bytes": float(per * case["records"] * case["passes"] + 32 * case["queries"]),
                "flops": 40.0 * case["records"] * case["passes"] + 60.0 * case["queries"]}
    if kind == "sdtree_query":
        return {"bytes": 60.0 * case["queries"], "flops": 120.0 * case["queries"]}
    if kind == "hashgrid":
        # both tables cleared, the current one copied to the previous one; positions in, slots out
        return {"bytes": 32.0 * case["slots"] + 16.0 * (case["points"] + case["queries"]),
                "flops": 20.0 * (case["points"] + case["queries"])}
    if kind == "trees":
        # per used cell the leaves read and cleared and the pyramid written; records and queries
        leaves, used = 4 ** case["level"], case["used"] * case["cells"]
        return {"bytes": used * (16.0 * leaves + 4.0 * (4 * leaves - 1) / 3) + (16.0 + 24.0) * case["queries"],
                "flops": used * leaves * 1.33 + 60.0 * case["queries"]}
    if kind == "mlp_train":
        f = 2.0 * (79 * 64 + 2 * 64 * 64 + 64 * 40)
        n = case["records"] * case["epochs"]
        return {"bytes": 52.0 * n + 8.0 * 16384, "flops": n * (3.0 * f - 2.0 * 79 * 64)}
    if kind == "mlp_eval":
        return {"bytes": (36.0 + (192.0 if case["raw"] else 160.0)) * case["samples"],
                "flops": 2.0 * (79 * 64 + 2 * 64 * 64 + 64 * 40) * case["samples"]}
    tris = case["objects"] * 20 * 4 ** case["level"]
    return {"bytes": (24.0 + 4 + 4 + 8 + 24 + 4 + 1) * case["rays"] + 112.0 * tris, "flops": 2 * case["rays"] * _ray_flops(tris)}


# ------------------------------------------------------------------ 64-bit results
def _net(params):
    w, o, out = torch.from_numpy(params.astype(np.float64)).to(DEV), 0, []
    for a, b in ((80, 64), (64, 64), (64, 64), (64, 48)):
        out.append(w[o:o + a * b].view(a, b).clone())
        o += a * b
    return out


def _forward(W, pos, nrm, wo):
    u = pos.double() / 10.0
    k = math.pi * 2.0 ** torch.arange(12, device=DEV, dtype=torch.float64)
    a = u[:, :, None] * k
    sc = torch.stack([torch.sin(a), torch.cos(a)], 3).reshape(len(u), 72)
    one = torch.ones((len(u), 1), device=DEV, dtype=torch.float64)
    h = torch.cat([sc, nrm.double(), wo.double(), one, 0 * one], 1)
    for l in range(3):
        h = torch.relu(h @ W[l])
    return h @ W[3]


def _lobes(raw):
    o = raw[:, :40].reshape(-1, 8, 5)
    mu = o[:, :, :3] / o[:, :, :3].norm(dim=2, keepdim=True).clamp_min(1e-12)
    return mu, torch.exp(o[:, :, 3].clamp(-2.3, 6.9)), torch.softmax(o[:, :, 4], 1)


def _exact_train(case, params, records):
    pos, nrm, wo, wi, w = records
    W = [p.requires_grad_(True) for p in _net(params)]
    m, v = [torch.zeros_like(p) for p in W], [torch.zeros_like(p) for p in W]
    t = loss = 0
    for _ in range(case["epochs"]):
        for b in range(0, case["records"], case["batch"]):
            i = slice(b, min(b + case["batch"], case["records"]))
            wt = w[i].double()
            total = wt.sum()
            wt = wt.clamp_max(20.0 * total / len(wt))
            mu, ka, al = _lobes(_forward(W, pos[i], nrm[i], wo[i]))
            f = ka / (2 * math.pi * (1 - torch.exp(-2 * ka))) * torch.exp(ka * ((mu * wi[i].double()[:, None]).sum(2) - 1))
            loss = -(wt * torch.log((al * f).sum(1).clamp_min(1e-30))).sum() / total
            grads = torch.autograd.grad(loss, W)
            t += 1
            with torch.no_grad():
                for k, g in enumerate(grads):
                    m[k] = 0.9 * m[k] + 0.1 * g
                    v[k] = 0.999 * v[k] + 0.001 * g * g
                    W[k] -= 1e-3 * (m[k] / (1 - 0.9 ** t)) / (torch.sqrt(v[k] / (1 - 0.999 ** t)) + 1e-8)
    return {"params": torch.cat([p.detach().reshape(-1) for p in W]).cpu().numpy(), "loss": float(loss)}


def _exact_hits(case, seed):
    tri = torch.from_numpy(np.ascontiguousarray(_rooms(case["objects"], case["lights"], case["level"])["tri_v"])).to(DEV)
    if case["rays"] * len(tri) > 4e9:
        return None
    org, d = (x.double() for x in _rays(case, seed, tri))
    v = tri.double().view(-1, 3, 3)
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    nn = (nrm * nrm).sum(1, keepdim=True)
    r0, r1, r2 = torch.linalg.cross(e2, nrm) / nn, torch.linalg.cross(nrm, e1) / nn, nrm / nn
    w0, w1, w2 = (-(r * v[:, 0]).sum(1) for r in (r0, r1, r2))
    out = torch.empty(case["rays"], device=DEV, dtype=torch.float64)
    step = max(1, int(6e7 // len(tri)))
    for a in range(0, case["rays"], step):
        o, q = org[a:a + step], d[a:a + step]
        t = -(o @ r2.T + w2) / (q @ r2.T)
        u, x = o @ r0.T + w0 + t * (q @ r0.T), o @ r1.T + w1 + t * (q @ r1.T)
        t = torch.where((t > 0) & (t < 1e20) & (u >= 0) & (x >= 0) & (u + x <= 1), t, math.inf).min(1).values
        out[a:a + step] = torch.where(torch.isinf(t), -torch.ones_like(t), t)
    return {"t": out, "prim": None, "uv": None, "occluded": None}


def exact(case, seed):
    """Network outputs, trained parameters and hit distances in 64 bits.  Renders, their
    gradients and guided samples have no such value: they are estimates whose paths follow
    single-precision decisions, and the guides' sums are integers."""
    g = _gen(seed)
    if case["kind"] == "mlp_eval":
        raw = _forward(_net(_weights(seed)), *_shading_points(case["samples"], g))
        if case["raw"]:
            return raw
        mu, ka, al = _lobes(raw)
        return torch.cat([mu, ka[..., None], al[..., None]], 2).reshape(-1, 40)
    if case["kind"] == "mlp_train":
        n = case["records"]
        pts = _shading_points(n, g)
        return _exact_train(case, _weights(seed), pts + (_vmf4(n, g), _lognormal(n, g)))
    if case["kind"] == "hits":
        return _exact_hits(case, seed)
    return None
