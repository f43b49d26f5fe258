"""The work that users of nan_b200 have it do, as cases that can be timed and
compared: the screen, texel and probe tracers, many probe sets in one batch,
the learned cache's inference and training, the consumers of the caches, the
visibility caster, scene builds and probe placement.

Scenes and sizes are those of the repository's benchmark and evaluation
programs (bench.py, benchmarks/) and tests; every scene is a seeded synthetic
one from nan_b200.scenes. `listed()` gives the cases, `draw()` more of the
same ranges, `prepare()` what a program holds before the call, `run()` one
pass through the public entry points, `exact()` the result in 64 bits where
plain torch or numpy can give it.
"""

from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

import nan_b200
from nan_b200 import _native, scenes
from nan_b200.mesh_colors import MeshColorsLayout, layout_adjacency
from nan_b200.radiance_cache import LAYER_SHAPES, initial_parameters
from nan_b200.surface_probe_resources import SURFACE_PROBE_DTYPE, SURFACE_PROBE_INSTANCE_SHIFT
from nan_b200.surface_probe_sampler import SurfaceProbeSampler

GRID, BOXES = 313, 500  # the 200,688-triangle terrain of the benchmark


def listed() -> list:
    return [
        # the smallest interactive frame: the 36-triangle box at 256x256, 1 spp, accumulated
        {"name": "screen_cornell", "path": "screen", "scene": "cornell", "width": 256, "height": 256, "vertices": 4},
        # a full-screen frame over about a million triangles, the reference's 5 path vertices
        {"name": "screen_terrain", "path": "screen", "scene": "terrain", "grid": 699, "boxes": 2000, "width": 1920,
         "height": 1080, "vertices": 5},
        # one iteration over every texel of the benchmark's Mesh Colors layout: the largest pass
        {"name": "texels_terrain", "path": "texels", "grid": GRID, "boxes": BOXES, "density": 16.0, "samples": 1,
         "bounces": 3, "compensated": False},
        # one iteration of the probe baker over the default site count
        {"name": "probes_terrain", "path": "probes", "grid": GRID, "boxes": BOXES, "sites": 20480, "samples": 16,
         "bounces": 3, "compensated": False},
        # probe sets of many scenes of uneven size in one batch, one random stream per sample
        {"name": "batch_probes", "path": "batch", "scenes": 16, "samples": 64, "bounces": 3, "independent": True,
         "wavefront": True},
        # the learned cache's answer for every pixel of a 1920x1080 frame
        {"name": "cache_infer", "path": "infer", "count": 1920 * 1080, "log2_table": 19},
        # one optimizer step of the learned cache on a batch of path vertices
        {"name": "cache_train", "path": "train", "count": 16384, "log2_table": 19, "update": "lazy"},
        # one surface-filter pass over the benchmark's texel cache
        {"name": "filter_terrain", "path": "filter", "grid": GRID, "boxes": BOXES, "density": 16.0},
        # a full-screen frame lit by the probe field
        {"name": "probe_resolve", "path": "resolve", "grid": GRID, "boxes": BOXES, "sites": 20480, "width": 1920,
         "height": 1080},
        # per-vertex visibility: the reference caster's 512 rays at every surface site
        {"name": "visibility", "path": "visibility", "grid": GRID, "boxes": BOXES, "sites": 65536, "rays": 512,
         "distance": 1000.0},
        # a scene rebuilt after its geometry changed
        {"name": "build_terrain", "path": "build", "grid": GRID, "boxes": BOXES},
        # probe placement: candidates thinned to a fifth by the adaptive elimination
        {"name": "place_adaptive", "path": "place", "candidates": 102400, "adaptive": True},
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    path = rng.choice(["screen", "screen", "texels", "texels", "probes", "batch", "infer", "train", "filter",
                       "resolve", "visibility", "build", "place"])
    land = {"grid": _log(rng, 20, 480), "boxes": _log(rng, 1, 800)}
    if path == "screen":
        size = {"width": _log(rng, 64, 1920), "height": _log(rng, 48, 1080), "vertices": rng.randint(2, 6)}
        if rng.random() < 0.4:
            return {"path": path, "scene": "cornell", **size}
        return {"path": path, "scene": "terrain", **land, **size}
    if path == "texels":
        land["grid"] = min(land["grid"], GRID)
        land["boxes"] = min(land["boxes"], BOXES)
        density = round(math.exp(rng.uniform(math.log(1.0), math.log(12.0))), 2)
        return {"path": path, **land, "density": density, "samples": rng.choice([1, 1, 2]),
                "bounces": rng.randint(1, 3), "compensated": rng.random() < 0.5}
    if path == "probes":
        return {"path": path, **land, "sites": _log(rng, 300, 40000), "samples": _log(rng, 1, 32),
                "bounces": rng.randint(1, 4), "compensated": rng.random() < 0.5}
    if path == "batch":
        return {"path": path, "scenes": rng.randint(2, 14), "samples": _log(rng, 4, 64), "bounces": rng.randint(1, 3),
                "independent": rng.random() < 0.6, "wavefront": rng.random() < 0.6}
    if path == "infer":
        return {"path": path, "count": _log(rng, 500, 2000000), "log2_table": rng.choice([14, 17, 19])}
    if path == "train":
        return {"path": path, "count": _log(rng, 1000, 65536), "log2_table": rng.choice([14, 17, 19]),
                "update": rng.choice(["lazy", "dense"])}
    if path == "filter":
        land["grid"] = min(land["grid"], GRID)
        land["boxes"] = min(land["boxes"], BOXES)
        return {"path": path, **land, "density": round(math.exp(rng.uniform(math.log(1.0), math.log(15.0))), 2)}
    if path == "resolve":
        return {"path": path, **land, "sites": _log(rng, 1000, 40000), "width": _log(rng, 160, 1920),
                "height": _log(rng, 90, 1080)}
    if path == "visibility":
        return {"path": path, **land, "sites": _log(rng, 100, 60000), "rays": rng.choice([64, 200, 512]),
                "distance": rng.choice([0.5, 20.0, 1000.0])}
    if path == "build":
        return {"path": path, **land}
    return {"path": path, "candidates": _log(rng, 2000, 200000), "adaptive": rng.random() < 0.5}


@functools.lru_cache(maxsize=1)
def _device():
    return nan_b200.Device(0)


def _terrain(case, seed):
    return scenes.terrain_boxes(seed=seed, grid=case["grid"], boxes=case["boxes"])


def _land_layout(node, case):
    return MeshColorsLayout.build(node, texels_per_unit=case["density"], min_resolution=4, max_resolution=64)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _surface_points(triangles, count, seed):
    """Area-weighted points of a scene's world triangles: (flat triangle,
    barycentrics of v1 and v2, positions, unit normals)."""
    t = triangles.cpu().numpy().reshape(-1, 3, 3)
    rng = np.random.default_rng(seed)
    n = np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    cdf = np.cumsum(np.linalg.norm(n.astype(np.float64), axis=1))
    flat = np.searchsorted(cdf, rng.random(count) * cdf[-1], side="right").clip(max=t.shape[0] - 1)
    u = rng.random((count, 2)).astype(np.float32)
    su = np.sqrt(u[:, :1])
    b1, b2 = (1 - u[:, 1:]) * su, u[:, 1:] * su
    p = (1 - b1 - b2) * t[flat, 0] + b1 * t[flat, 1] + b2 * t[flat, 2]
    n = n[flat] / np.linalg.norm(n[flat], axis=1, keepdims=True)
    return flat, np.concatenate([b1, b2], 1), p, n


def _site_layout(node, scene, count, seed):
    """Probe sites on the scene's surfaces, packed with their octrees."""
    flat, b, p, n = _surface_points(scene.world_triangles(), count, seed)
    first = np.concatenate([[0], np.cumsum([node.meshes[m].indices.shape[0] for m, _, _ in node.instances])])
    inst = np.searchsorted(first, flat, side="right") - 1
    order = np.argsort(inst, kind="stable")
    r = np.zeros(count, dtype=SURFACE_PROBE_DTYPE)
    r["position_radius"][:, :3] = p[order]
    r["normal_side"][:, :3] = n[order]
    r["normal_side"][:, 3] = 1.0
    r["meta"][:, 0] = (flat - first[inst])[order]
    r["meta"][:, 1] = np.ascontiguousarray(b[order, 0]).view(np.uint32)
    r["meta"][:, 2] = np.ascontiguousarray(b[order, 1]).view(np.uint32)
    r["meta"][:, 3] = (inst[order] << SURFACE_PROBE_INSTANCE_SHIFT).astype(np.uint32)
    return nan_b200.SurfaceProbeSiteLayout.from_sites(node, r, sampler=SurfaceProbeSampler(_device()))


def _baker(node, case, sites, seed, compensated=True):
    dev = _device()
    scene = nan_b200.Scene(dev, node)
    geometry = nan_b200.SurfaceProbeGpuGeometry.create(dev, _site_layout(node, scene, sites, seed))
    baker = nan_b200.SurfaceProbeDiffuseIrradianceBaker(dev, scene, geometry, samples_per_probe=case["samples"],
                                                        max_bounces=case["bounces"], compensated=compensated)
    rt = nan_b200.SurfaceProbeRuntimeBuffers.acquire(nan_b200.RenderData(dev), geometry.probe_count)
    return baker, rt


def _probe_outputs(rt):
    return [rt.field.values.view(torch.float32), rt.field.sample_counts.view(torch.int32),
            rt.attachments.self_hit_counts.view(torch.int32), rt.attachments.radial_moments.view(torch.float16)]


def _slot_count(case, layout) -> int:
    """Slots of the buffers a program keeps: one size for the scenes of all
    seeds, whose layouts differ by a few per cent."""
    n = _texel_count(case["grid"], case["boxes"], case["density"])
    n += n // 4 + 4096
    if layout.total_payload_count > n:
        raise ValueError("layout larger than the slot buffers")
    return n


def _irradiance_slots(payload, seed):
    g = _generator(seed)
    slots = torch.empty((payload, 4), dtype=torch.float32, device="cuda")
    slots[:, :3] = torch.rand((payload, 3), device="cuda", generator=g) * 3.0
    slots[:, 3] = torch.randint(1, 64, (payload,), device="cuda", generator=g, dtype=torch.int32).view(torch.float32)
    return slots


def _cache_inputs(case, seed):
    """Parameters of trained size, queries in the order of a frame's pixels (a
    first hit moves with the pixel over a rolling terrain, the queried second
    hit lies some way off it), and irradiance targets."""
    g = _generator(seed)
    n = case["count"]
    mlp, _ = initial_parameters(10, seed)
    table = (torch.rand(16 * 2 << case["log2_table"], device="cuda", generator=g) - 0.5) * 0.4
    q = torch.zeros((n, 8), device="cuda")
    i, wide = torch.arange(n, device="cuda"), max(1, math.isqrt(16 * n // 9))
    if case["path"] == "train":  # training points are strided over the frame
        i = (i * 617) % n
    away = torch.randn((n, 2), device="cuda", generator=g) * 0.04
    q[:, 0] = ((i % wide) / wide + away[:, 0]).clamp(0.0, 1.0)
    q[:, 2] = ((i // wide) * wide / n + away[:, 1]).clamp(0.0, 1.0)
    q[:, 1] = 0.4 + 0.2 * torch.sin(6.0 * q[:, 0]) * torch.cos(5.0 * q[:, 2])
    q[:, 4:7] = torch.nn.functional.normalize(torch.randn((n, 3), device="cuda", generator=g), dim=1)
    y = torch.zeros((n, 4), device="cuda")
    y[:, :3] = torch.rand((n, 3), device="cuda", generator=g) * 3.0
    return torch.from_numpy(mlp).cuda(), table, q, y


def _batch_sizes(count):
    """(grid, boxes, sites) of each scene: triangles spread over 1e3..5e5 on a
    log scale, 95 % of them terrain, and 512..20480 sites, in mixed order."""
    out = []
    for i in range(count):
        t = math.exp(math.log(1e3) + math.log(5e2) * (i + 0.5) / count)
        out.append((max(3, int(round(math.sqrt(0.475 * t))) + 1), max(1, int(0.05 * t / 12.0)),
                    512 + (i * 7919 + 6151) % 19969))
    return out[1::2] + out[::2]


def prepare(case, seed):
    dev = _device()
    path = case["path"]
    if path == "screen":
        if case["scene"] == "cornell":
            node = scenes.cornell_box(case["width"], case["height"])
        else:
            node = _terrain(case, seed)
        scene = nan_b200.Scene(dev, node)
        out = torch.zeros((case["height"], case["width"], 4), device="cuda")
        return {"path": path, "tracer": nan_b200.PathTracer(dev, scene, max_vertices=case["vertices"]),
                "accumulator": nan_b200.Accumulator(dev), "rd": nan_b200.RenderData(dev), "camera": scene.camera,
                "out": out, "display": torch.zeros_like(out), "frame": seed % 65536}
    if path == "texels":
        node = _terrain(case, seed)
        layout = _land_layout(node, case)
        tracer = nan_b200.TextureSpacePathTracer(dev, nan_b200.Scene(dev, node), layout,
                                                 samples_per_texel=case["samples"], max_bounces=case["bounces"],
                                                 compensated=case["compensated"])
        slots = torch.zeros((_slot_count(case, layout), 4), dtype=torch.int32, device="cuda")
        return {"path": path, "tracer": tracer, "slots": slots, "iteration": 0}
    if path == "probes":
        baker, rt = _baker(_terrain(case, seed), case, case["sites"], seed, case["compensated"])
        return {"path": path, "baker": baker, "rt": rt, "iteration": 0}
    if path == "batch":
        items = [_baker(scenes.terrain_boxes(seed=1000 * seed + i, grid=grid, boxes=boxes), case, sites, seed)
                 for i, (grid, boxes, sites) in enumerate(_batch_sizes(case["scenes"]))]
        batch = nan_b200.ProbeBatch(dev, [(b, rt.field, rt.attachments) for b, rt in items],
                                    independent_samples=case["independent"], wavefront=case["wavefront"])
        return {"path": path, "batch": batch, "rts": [rt for _, rt in items], "case": dict(case), "iteration": 0}
    if path in ("infer", "train"):
        mlp, table, q, y = _cache_inputs(case, seed)
        cache = nan_b200.RadianceCache(dev, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), log2_table=case["log2_table"],
                                       table_update=case.get("update", "dense"))
        cache.set_params(mlp, table)
        return {"path": path, "cache": cache, "queries": q, "targets": y}
    if path == "filter":
        node = _terrain(case, seed)
        layout = _land_layout(node, case)
        scene = nan_b200.Scene(dev, node)
        src = _irradiance_slots(_slot_count(case, layout), seed)
        return {"path": path, "filter": nan_b200.MeshColorsSurfaceFilter(dev, scene, layout), "src": src,
                "dst": torch.zeros_like(src)}
    if path == "resolve":
        node = _terrain(case, seed)
        scene = nan_b200.Scene(dev, node)
        layout = _site_layout(node, scene, case["sites"], seed)
        geometry = nan_b200.SurfaceProbeGpuGeometry.create(dev, layout)
        n = geometry.probe_count
        rt = nan_b200.SurfaceProbeRuntimeBuffers.acquire(nan_b200.RenderData(dev), n)
        g = _generator(seed + 1)
        rt.field.values.view(torch.float32).copy_(torch.rand(3 * n, device="cuda", generator=g) * 2.0 + 0.2)
        rt.field.sample_counts.view(torch.int32).copy_(
            torch.randint(1, 64, (n,), device="cuda", generator=g, dtype=torch.int32))
        mean = torch.rand(16 * n, device="cuda", generator=g) * 1.9 + 0.1
        moments = torch.stack([mean, mean * mean + 0.1 * torch.rand(16 * n, device="cuda", generator=g)], 1)
        rt.attachments.radial_moments.view(torch.float16).copy_(moments.half().reshape(-1))
        return {"path": path, "resolve": nan_b200.SurfaceProbeResolve(dev, scene, layout, geometry), "rt": rt,
                "camera": scene.camera, "out": torch.zeros((case["height"], case["width"], 4), device="cuda")}
    if path == "visibility":
        node = _terrain(case, seed)
        scene = nan_b200.Scene(dev, node)
        _, _, p, n = _surface_points(scene.world_triangles(), case["sites"], seed)
        return {"path": path, "sampler": nan_b200.PMRVisibilitySHSampler(dev), "scene": scene,
                "positions": torch.from_numpy(p).cuda(), "normals": torch.from_numpy(n).cuda(), "rays": case["rays"],
                "distance": case["distance"]}
    if path == "build":
        packed = _terrain(case, seed).pack()
        buf = {k: torch.from_numpy(v.view(np.int32) if v.dtype == np.uint32 else v).cuda() for k, v in packed.items()}
        desc = _native.NanSceneDesc()
        for k in ("vertices", "indices", "mesh_descs", "instance_descs", "transforms", "inverse_transposes",
                  "materials"):
            setattr(desc, k, _native.ptr(buf[k]))
        desc.vertex_count, desc.index_triangle_count = packed["vertices"].shape[0], packed["indices"].shape[0]
        desc.mesh_count, desc.instance_count = packed["mesh_descs"].shape[0], packed["instance_descs"].shape[0]
        desc.transform_count, desc.material_count = packed["transforms"].shape[0], packed["materials"].shape[0]
        count = int((packed["mesh_descs"][:, 1][packed["instance_descs"][:, 0]] // 3).sum())
        g = _generator(seed)
        rays = torch.zeros((16384, 8), device="cuda")  # what a program asks of the new tree: who hits what
        rays[:, :3] = (torch.rand((16384, 3), device="cuda", generator=g) - 0.5) * 0.15 * case["grid"]
        rays[:, 1] = 3.0
        rays[:, 4:7] = torch.nn.functional.normalize(torch.randn((16384, 3), device="cuda", generator=g), dim=1)
        rays[:, 7] = 1000.0
        return {"path": path, "buffers": buf, "desc": desc, "context": dev.new_context(), "rays": rays,
                "triangles": torch.empty((count, 9), device="cuda"),
                "ids": torch.empty((16384, 4), dtype=torch.int32, device="cuda"),
                "hits": torch.empty((16384, 3), device="cuda")}
    if path == "place":
        p, n, d = _candidates(case, seed)
        return {"path": path, "sampler": SurfaceProbeSampler(dev), "positions": p, "normals": n,
                "densities": d if case["adaptive"] else None, "count": case["candidates"],
                "area": _place_area(case)}
    raise ValueError(path)


def _place_area(case) -> float:
    return case["candidates"] / 90.0  # candidates per square metre as in the placement evaluation


def _candidates(case, seed):
    """Candidates on a rolling height field of the stated area, with normals
    and densities that vary 6:1 across it."""
    g = _generator(seed)
    n = case["candidates"]
    side = math.sqrt(_place_area(case))
    x, z = (torch.rand(n, device="cuda", generator=g) * side for _ in range(2))
    p = torch.stack([x, 0.5 * torch.sin(0.9 * x) * torch.cos(0.7 * z), z], 1)
    dx = 0.45 * torch.cos(0.9 * x) * torch.cos(0.7 * z)
    dz = -0.35 * torch.sin(0.9 * x) * torch.sin(0.7 * z)
    nrm = torch.nn.functional.normalize(torch.stack([-dx, torch.ones_like(x), -dz], 1), dim=1)
    return p, nrm, 0.4 + 2.0 * (0.5 + 0.5 * torch.sin(0.7 * x + 0.3 * z))


def run(s):
    path = s["path"]
    if path == "screen":
        out, display = s["out"], s["display"]
        s["camera"].begin_frame(out.shape[1], out.shape[0])
        s["tracer"].execute(None, out, s["frame"])
        s["accumulator"].execute(None, s["rd"], out, display, reset=False)
        s["frame"] += 1
        return [out, display]
    if path == "texels":
        s["tracer"].execute(None, s["slots"], s["iteration"], reset=(s["iteration"] == 0))
        s["iteration"] += 1
        return [s["slots"].view(torch.float32)[:, :3], s["slots"][:, 3]]
    if path == "probes":
        rt = s["rt"]
        s["baker"].execute(None, rt.field, rt.attachments, s["iteration"], reset=(s["iteration"] == 0))
        s["iteration"] += 1
        return _probe_outputs(rt)
    if path == "batch":
        c = s["case"]
        s["batch"].execute(None, s["iteration"], c["samples"], c["bounces"], reset=(s["iteration"] == 0))
        s["iteration"] += 1
        return [_probe_outputs(rt) for rt in s["rts"]]
    if path == "infer":
        return [s["cache"].infer(s["queries"])]
    if path == "train":
        cache = s["cache"]
        cache.backward(s["queries"], s["targets"])
        grads = cache.gradients()
        cache.step()
        return list(grads)
    if path == "filter":
        s["filter"].execute(None, s["src"], s["dst"])
        return [s["dst"][:, :3], s["dst"].view(torch.int32)[:, 3]]
    if path == "resolve":
        out, rt = s["out"], s["rt"]
        s["camera"].begin_frame(out.shape[1], out.shape[0])
        s["resolve"].execute(None, rt.field, rt.attachments, out)
        return [out]
    if path == "visibility":
        sh = s["sampler"].sample(s["scene"], s["positions"], s["normals"], ray_count=s["rays"],
                                 max_distance=s["distance"])
        return [sh, s["sampler"].visible_counts]
    if path == "build":
        lib, handle, stream = _native.lib(), s["context"].handle, _native.stream_handle(None)
        _native.check(lib.nan_scene_build(handle, ctypes.byref(s["desc"]), stream))
        _native.check(lib.nan_scene_world_triangles(handle, _native.ptr(s["triangles"]), stream))
        _native.check(lib.nan_intersect(handle, _native.ptr(s["rays"]), s["rays"].shape[0], _native.ptr(s["ids"]),
                                        _native.ptr(s["hits"]), stream))
        return [s["triangles"], s["ids"], s["hits"]]
    n = s["count"]
    keep, radii = s["sampler"].eliminate(s["positions"], s["normals"], [0, n], [n // 5], [s["area"]],
                                         relative_densities=s["densities"])
    return [keep, radii]


# ---------------------------------------------------------------------------
# Bytes and operations that a pass cannot do without.
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _texel_count(grid, boxes, density) -> int:
    node = scenes.terrain_boxes(seed=1, grid=grid, boxes=boxes)
    return MeshColorsLayout.build(node, texels_per_unit=density, min_resolution=4,
                                  max_resolution=64).total_surface_texels


def _triangles(case) -> int:
    return 36 if case.get("scene") == "cornell" else 2 * (case["grid"] - 1) ** 2 + 12 * case["boxes"]


def _ray_flops(triangles) -> float:
    """One descent of a binary tree over the triangles (two boxes of 12
    operations a level) and two triangle tests of 50."""
    return 24.0 * math.log2(max(triangles, 2)) + 100.0


def work(case) -> dict:
    path = case["path"]
    if path == "screen":
        px, tri = case["width"] * case["height"], _triangles(case)
        return {"bytes": 64.0 * px + 96.0 * tri, "flops": px * 2.0 * _ray_flops(tri)}
    if path == "texels":
        n, tri = _texel_count(case["grid"], case["boxes"], case["density"]), _triangles(case)
        slot = 64.0 if case["compensated"] else 32.0
        return {"bytes": slot * n + 96.0 * tri, "flops": 3.0 * n * case["samples"] * _ray_flops(tri)}
    if path == "probes":
        n, tri = case["sites"], _triangles(case)
        return {"bytes": 200.0 * n + 96.0 * tri, "flops": 2.0 * n * case["samples"] * _ray_flops(tri)}
    if path == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for grid, boxes, sites in _batch_sizes(case["scenes"]):
            tri = _triangles({"grid": grid, "boxes": boxes})
            total["bytes"] += 200.0 * sites + 96.0 * tri
            total["flops"] += 2.0 * sites * case["samples"] * _ray_flops(tri)
        return total
    mlp = 2.0 * sum(r * c for r, c in LAYER_SHAPES)
    table = 4.0 * 16 * 2 ** case.get("log2_table", 0)
    if path == "infer":
        return {"bytes": 48.0 * case["count"] + min(table, 512.0 * case["count"]), "flops": mlp * case["count"]}
    if path == "train":
        # queries, targets and touched entries once; the gradients that come back whole
        return {"bytes": 48.0 * case["count"] + 2.0 * table, "flops": 3.0 * mlp * case["count"]}
    if path == "filter":
        n = _texel_count(case["grid"], case["boxes"], case["density"])
        return {"bytes": 32.0 * n + 32.0 * _triangles(case), "flops": 50.0 * n}
    if path == "resolve":
        px, tri = case["width"] * case["height"], _triangles(case)
        return {"bytes": 16.0 * px + 96.0 * tri + 140.0 * case["sites"],
                "flops": px * (2.0 * _ray_flops(tri) + 20 * 100.0)}
    if path == "visibility":
        tri = _triangles(case)
        return {"bytes": 92.0 * case["sites"] + 96.0 * tri,
                "flops": 1.0 * case["sites"] * case["rays"] * _ray_flops(tri)}
    if path == "build":
        tri = _triangles(case)
        return {"bytes": 160.0 * tri, "flops": 100.0 * tri}
    return {"bytes": 29.0 * case["candidates"], "flops": 18 * 30.0 * case["candidates"]}


# ---------------------------------------------------------------------------
# The same in 64 bits, by plain torch and numpy.
# ---------------------------------------------------------------------------
def exact(case, seed):
    path = case["path"]
    if path == "screen" and case["scene"] == "cornell":
        img = _exact_box_frame(case, seed)
        return [img, img]
    if path == "infer":
        mlp, table, q, _ = _cache_inputs(case, seed)
        out = torch.zeros((case["count"], 4), dtype=torch.float64, device="cuda")
        with torch.no_grad():
            for a in range(0, case["count"], 1 << 18):
                out[a:a + (1 << 18), :3] = _exact_network(case, mlp.double(), table.double(), q[a:a + (1 << 18)])
        return [out]
    if path == "train":
        mlp, table, q, y = _cache_inputs(case, seed)
        w = mlp.double().requires_grad_(True)
        t = table.double().requires_grad_(True)
        o = _exact_network(case, w, t, q)
        loss = ((o - y[:, :3].double()) ** 2 / (o.detach() ** 2 + float(np.float32(1e-2)))).sum() / case["count"]
        loss.backward()
        return [w.grad, t.grad, loss.detach().reshape(1)]
    if path == "filter":
        node = _terrain(case, seed)
        return [_exact_filter(case, node, _land_layout(node, case), seed), None]
    if path == "build":
        return [_exact_world(_terrain(case, seed)), None, None]
    if path == "place":
        r = math.sqrt(np.float32(_place_area(case)) / (2.0 * math.sqrt(3.0) * (case["candidates"] // 5)))
        return [None, np.array([r])]
    # random walks over scenes of many triangles: no quick form without a tree
    return None


def _exact_world(node):
    rows = []
    for mesh_id, _, transform_id in node.instances:
        mesh, m = node.meshes[mesh_id], node.transforms[transform_id].astype(np.float64)
        p = mesh.vertices[:, :3].astype(np.float64) @ m[:3, :3].T + m[:3, 3]
        rows.append(p[mesh.indices.astype(np.int64)].reshape(-1, 9))
    return np.concatenate(rows)


def _exact_network(case, mlp, table, q):
    """Hash encoding (Mueller et al. 2022) and ReLU network, in 64 bits."""
    p, size = q[:, :3].double().clamp(0.0, 1.0), 1 << case["log2_table"]
    growth = math.exp((math.log(2048) - math.log(16)) / 15)
    table = table.view(16, size, 2)
    feats = []
    for level in range(16):
        r = math.floor(16 * growth ** level)
        s = p * r
        c = s.floor().clamp(max=r - 1)
        f, ci = s - c, c.long()
        acc = 0.0
        for k in range(8):
            d = [(k >> a) & 1 for a in range(3)]
            g = [ci[:, a] + d[a] for a in range(3)]
            if (r + 1) ** 3 <= size:
                idx = g[0] + g[1] * (r + 1) + g[2] * (r + 1) ** 2
            else:
                idx = (g[0] ^ (g[1] * 2654435761) ^ (g[2] * 805459861)) & (size - 1)
            w = 1.0
            for a in range(3):
                w = w * (f[:, a] if d[a] else 1.0 - f[:, a])
            acc = acc + w[:, None] * table[level][idx & (size - 1)]
        feats.append(acc)
    n = q.shape[0]
    one = torch.ones((n, 1), dtype=torch.float64, device=q.device)
    x = torch.cat(feats + [q[:, 4:7].double(), one, torch.zeros((n, 12), dtype=torch.float64, device=q.device)], 1)
    off = 0
    for i, (rows, cols) in enumerate(LAYER_SHAPES):
        x = x @ mlp[off:off + rows * cols].view(rows, cols).t()
        off += rows * cols
        if i < 4:
            x = x.relu()
    return x[:, :3]


def _exact_filter(case, node, layout, seed):
    """One filter pass (spatial sigma 1, normal sigma 30 degrees) over a
    scene without double-sided materials."""
    dev = "cuda"
    src = _irradiance_slots(_slot_count(case, layout), seed)[:, :3].double()
    tri = torch.from_numpy(_exact_world(node)).to(dev).view(-1, 3, 3)
    nrm = torch.nn.functional.normalize(torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]), dim=1)
    inst = torch.from_numpy(layout.instance_array.astype(np.int64)).to(dev)
    faces = torch.from_numpy(layout.face_array.astype(np.int64)).to(dev)
    adjacency = torch.from_numpy(layout_adjacency(node).astype(np.int64)).to(dev)
    inst_of_face = torch.repeat_interleave(torch.arange(inst.shape[0], device=dev), inst[:, 1])
    base = faces[:, 0] + inst[inst_of_face, 2]
    res = faces[:, 1]

    def slot(face, i, j):
        return base[face] + i * (res[face] + 1) - (i * (i - 1)).div(2, rounding_mode="floor") + j

    out = torch.zeros_like(src)
    weight = math.exp(-0.5)
    for r in torch.unique(res).tolist():
        ij = torch.tensor([(i, j) for i in range(r + 1) for j in range(r + 1 - i)], device=dev)
        which = torch.nonzero(res == r).flatten()
        step = max(1, (1 << 22) // ij.shape[0])
        for a in range(0, which.shape[0], step):
            part = which[a:a + step]
            f = part.repeat_interleave(ij.shape[0])
            i, j = ij[:, 0].repeat(part.shape[0]), ij[:, 1].repeat(part.shape[0])
            center = slot(f, i, j)
            acc = src[center].clone()
            total = torch.ones(acc.shape[0], dtype=torch.float64, device=dev)
            for dx, dy in ((1, 0), (-1, 0), (0, 1), (0, -1), (1, -1), (-1, 1)):
                x, y = i + dx, j + dy
                inside = (x >= 0) & (y >= 0) & (x + y <= r)
                k = torch.nonzero(inside).flatten()
                acc[k] += weight * src[slot(f[k], x[k], y[k])]
                total[k] += weight
                k = torch.nonzero(~inside).flatten()
                edge = torch.where(x[k] < 0, 1, torch.where(y[k] < 0, 2, 0))
                packed = adjacency[f[k], edge]
                ok = packed != 0xFFFFFFFF
                k, edge, packed = k[ok], edge[ok], packed[ok]
                g = inst[inst_of_face[f[k]], 0] + (packed >> 3)
                b = torch.stack([x[k], y[k], r - x[k] - y[k]], 1).double() / r
                rows = torch.arange(k.shape[0], device=dev)
                outside = b[rows, (edge + 2) % 3]
                start, flip = packed & 3, (packed & 4) != 0
                end, opposite = (start + 1) % 3, (start + 2) % 3
                nb = torch.zeros_like(b)
                nb[rows, torch.where(flip, end, start)] = b[rows, edge] + outside
                nb[rows, torch.where(flip, start, end)] = b[rows, (edge + 1) % 3] + outside
                nb[rows, opposite] = -outside
                ok = ((nb >= -1e-5) & (nb <= 1 + 1e-5)).all(1)
                k, g, nb = k[ok], g[ok], nb[ok].clamp(min=0.0)
                nb = nb / nb.sum(1, keepdim=True)
                cosine = (nrm[f[k]] * nrm[g]).sum(1).clamp(0.0, 1.0)
                w = weight * torch.exp(-0.5 * (torch.acos(cosine) / math.radians(30.0)) ** 2)
                # linear interpolation on the lattice cell that holds the point
                s = nb * res[g][:, None]
                s = torch.where((s - s.round()).abs() < 1e-9, s.round(), s)
                c0 = torch.minimum(s[:, 0].floor().long(), res[g])
                c1 = torch.minimum(s[:, 1].floor().long(), res[g] - c0)
                u = s - s.floor()
                upper = (u.sum(1) - 2.0).abs() <= 1e-3
                u = torch.where(upper[:, None], 1.0 - u, u)
                corner = (u.sum(1) <= 1e-6) | (c0 + c1 >= res[g])
                up = upper.long()
                lim = torch.where(corner, 0, 1)
                va = src[slot(g, c0 + lim * (1 - up), c1 + lim * up)]
                vb = src[slot(g, c0 + lim * up, c1 + lim * (1 - up))]
                vc = src[slot(g, c0 + lim * up, c1 + lim * up)]
                v = u[:, :1] * va + u[:, 1:2] * vb + u[:, 2:] * vc
                v = torch.where(corner[:, None], src[slot(g, c0, c1)], v)
                acc[k] += w[:, None] * v
                total[k] += w
            out[center] = acc / total[:, None]
    return out


def _exact_box_frame(case, seed):
    """The first frame of the 36-triangle box (lit by its ceiling quad alone):
    every path by brute force over the triangles, with the tracer's random
    streams (an LCG per pixel and frame)."""
    dev, w, h = "cuda", case["width"], case["height"]
    node = scenes.cornell_box(w, h)
    f64 = {"dtype": torch.float64, "device": dev}
    tri = torch.from_numpy(_exact_world(node)).to(dev).view(-1, 3, 3)
    mats = [node.materials[m] for me, m, _ in node.instances for _ in range(node.meshes[me].indices.shape[0])]
    albedo = torch.tensor(np.array([m.base_color for m in mats], np.float32), device=dev).double()
    emission = torch.tensor(np.array([m.emissive for m in mats], np.float32), device=dev).double()
    two_sided = torch.tensor([bool(m.double_sided) for m in mats], device=dev)
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    normal = torch.nn.functional.normalize(torch.linalg.cross(e1, e2), dim=1)

    cam = node.camera
    pos = torch.tensor(np.asarray(cam.position, np.float64), device=dev)
    fwd = torch.nn.functional.normalize(torch.tensor(np.asarray(cam.target, np.float64), device=dev) - pos, dim=0)
    right = torch.nn.functional.normalize(torch.linalg.cross(fwd, torch.tensor([0.0, 1.0, 0.0], **f64)), dim=0)
    up = torch.linalg.cross(right, fwd)
    half = math.tan(math.radians(cam.fov) * 0.5)
    py, px = torch.meshgrid(torch.arange(h, device=dev), torch.arange(w, device=dev), indexing="ij")
    px, py = px.reshape(-1), py.reshape(-1)
    nx, ny = 2.0 * (px.double() + 0.5) / w - 1.0, 1.0 - 2.0 * (py.double() + 0.5) / h
    d = fwd + nx[:, None] * right * (half * w / h) + ny[:, None] * up * half
    d = torch.nn.functional.normalize(d, dim=1)
    o = pos.expand_as(d)

    state = (px * 100591) ^ (py * 102191) ^ ((seed % 65536) * 103643) & 0xFFFFFFFF
    state = state & 0xFFFFFFFF

    def uniform():
        nonlocal state
        state = (1664525 * state + 1013904223) & 0xFFFFFFFF
        return (state >> 8).double() * 2.0 ** -24

    uniform(), uniform()
    light = torch.zeros_like(d)
    through = torch.ones_like(d)
    alive = torch.ones(d.shape[0], dtype=torch.bool, device=dev)
    for _ in range(case["vertices"]):
        best = torch.full((d.shape[0],), 1000.0, **f64)
        hit = torch.full((d.shape[0],), -1, device=dev)
        for k in range(tri.shape[0]):
            pv = torch.linalg.cross(d, e2[k].expand_as(d))
            det = (pv * e1[k]).sum(1)
            s = o - tri[k, 0]
            qv = torch.linalg.cross(s, e1[k].expand_as(s))
            u, v, t = (pv * s).sum(1) / det, (d * qv).sum(1) / det, (qv * e2[k]).sum(1) / det
            ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 1e-5) & (t < best)
            best, hit = torch.where(ok, t, best), torch.where(ok, k, hit)
        alive = alive & (hit >= 0)
        at = hit.clamp(min=0)
        n = normal[at]
        back = two_sided[at] & ((n * d).sum(1) >= 0)
        n = torch.where(back[:, None], -n, n)
        light = light + torch.where(alive[:, None], through * emission[at], 0.0)
        uniform(), uniform()  # the sun's sample: no sun shines here
        a, b = uniform(), uniform()
        cos = b.sqrt()
        sin = (1.0 - cos * cos).clamp(min=0.0).sqrt()
        phi = 2.0 * math.pi * a
        tan = torch.nn.functional.normalize(
            torch.linalg.cross(n, torch.stack([-n[:, 2], n[:, 0], -n[:, 1]], 1)), dim=1)
        bit = torch.linalg.cross(n, tan)
        o = o + best[:, None] * d
        d = (sin * phi.cos())[:, None] * tan + (sin * phi.sin())[:, None] * bit + cos[:, None] * n
        through = through * albedo[at]
    img = torch.ones((h * w, 4), **f64)
    img[:, :3] = light
    return img.view(h, w, 4)
