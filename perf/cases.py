"""The framework's performance cases: whole calls of its public entry points.

Every case is one call, or one short sequence of calls, that a multi-view
stereo program makes: a depth map of one reference view
(``PatchMatchACMMCuda``), a batch of depth maps over resident views
(``DepthMapPool``), the cross-view filter of a cluster (``CrossFilterCuda``),
the fusion of its maps (``StereoFusion``), an initial map from a prior model
(``init_maps``) and the rescaling between pyramid levels (``pyramid``).

Scenes are seeded: a textured heightfield rendered by the package's ray-caster
from cameras around one pose, with the gain, noise, outliers and holes that the
images and maps of a real capture have. All inputs are on the GPU.
"""
import math

import numpy as np
import torch

from sensemap_b200 import STORE_F16, STORE_F32, STORE_U8
from sensemap_b200 import _native as native
from sensemap_b200 import init_maps, pyramid
from sensemap_b200 import synthetic as syn
from sensemap_b200.cross_filter import CrossFilterCuda, filter_problems
from sensemap_b200.fusion import FusionImage, FusionOptions, StereoFusion
from sensemap_b200.patch_match import PatchMatchACMMCuda, PatchMatchOptions, Problem, View
from sensemap_b200.pool import DepthMapPool

STORAGE = {"u8": STORE_U8, "f16": STORE_F16, "f32": STORE_F32}
WINDOWS = [(5, 2), (5, 1), (3, 1), (3, 2), (4, 2), (7, 2)]  # (radius, step)


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def depth_map(name, width, height, sources, radius, step, iterations, storage, mode):
    c = {"kind": "depth_map", "width": width, "height": height, "sources": sources, "radius": radius, "step": step,
         "iterations": iterations, "storage": storage, "mode": mode}
    return dict(c, name=name) if name else c


def listed():
    return [
        # A thumbnail-sized map, as a preview or the coarsest pyramid level asks for: launches and set-up count.
        depth_map("depth map 160x120", 160, 120, 4, 5, 2, 5, "u8", "photometric"),
        # The 640x480 planes configuration: 1 + 4 views, plain FP32 sources, every tap of the window.
        depth_map("depth map 640x480", 640, 480, 4, 5, 1, 6, "f32", "photometric"),
        # The headline configuration: 1600x1200, 10 sources, FP16 sources, every tap of the window.
        depth_map("depth map 1600x1200", 1600, 1200, 10, 5, 1, 6, "f16", "photometric"),
        # The default options (window step 2, 5 iterations, 8-bit sources, geometric term) at odd sizes.
        depth_map("geometric map 1201x899", 1201, 899, 8, 5, 2, 5, "u8", "geometric"),
        # A fine pyramid level of a large view: 20 sources, 3 iterations from the coarser level's maps.
        depth_map("geometric map 3000x2000", 3000, 2000, 20, 5, 2, 3, "f16", "geometric"),
        # A batch of references of uneven size and source count over resident views, in one pool.
        {"name": "pool of 6 jobs", "kind": "pool", "jobs": 6, "width": 1200, "height": 900, "radius": 5, "step": 2,
         "iterations": 5},
        # The cross-view filter and deduplication of a cluster of 11 views, maps staying on the GPU.
        {"name": "cross filter 11x1600x1200", "kind": "cross_filter", "views": 11, "width": 1600, "height": 1200,
         "host": False},
        # The same for a small cluster at odd sizes, its maps read back.
        {"name": "cross filter 5x401x301", "kind": "cross_filter", "views": 5, "width": 401, "height": 301,
         "host": True},
        # The fusion of a cluster's maps into a point cloud.
        {"name": "fusion 11x1600x1200", "kind": "fusion", "views": 11, "width": 1600, "height": 1200,
         "clean": False},
        # A small cluster's fusion with both clean-up passes.
        {"name": "fusion 6x640x480", "kind": "fusion", "views": 6, "width": 640, "height": 480, "clean": True},
        # The initial map of a view from an oriented point cloud.
        {"name": "initial map 1600x1200", "kind": "initial_map", "source": "dense", "width": 1600, "height": 1200,
         "points": 400000},
        # One view's image taken to two coarser levels and its maps carried back to full size.
        {"name": "pyramid 3000x2000", "kind": "pyramid", "width": 3000, "height": 2000, "levels": 3},
    ]


def _between(rng, lo, hi):
    """A whole number from lo to hi, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["depth_map"] * 5 + ["pool"] + ["cross_filter"] * 2 + ["fusion"] * 2 +
                      ["initial_map"] * 2 + ["pyramid"])
    aspect = rng.uniform(0.6, 0.85)
    if kind == "depth_map":
        radius, step = rng.choice(WINDOWS)
        mode = rng.choice(["photometric", "geometric"])
        c = depth_map(None, _between(rng, 120, 3000), 0, _between(rng, 2, 20), radius, step,
                      rng.randint(3, 6), rng.choice(list(STORAGE)), mode)
        c["height"] = max(90, int(c["width"] * aspect))
        while work(c)["flops"] > 2.5e12:  # at most about half of the largest listed case
            c["width"], c["height"] = int(c["width"] * 0.8), max(90, int(c["height"] * 0.8))
        return c
    if kind == "pool":
        width = _between(rng, 240, 1200)
        return {"kind": "pool", "jobs": rng.randint(2, 6), "width": width, "height": int(width * aspect),
                "radius": 5, "step": rng.choice([1, 2]) if width < 700 else 2, "iterations": rng.randint(3, 5)}
    if kind in ("cross_filter", "fusion"):
        width = _between(rng, 200, 1600)
        c = {"kind": kind, "views": rng.randint(4, 11), "width": width, "height": int(width * min(aspect, 0.75))}
        if kind == "fusion":
            return dict(c, clean=rng.random() < 0.5)
        return dict(c, host=width < 500)
    if kind == "initial_map":
        width = _between(rng, 320, 1600)
        source = rng.choice(["sparse", "mesh", "dense", "delaunay"])
        return {"kind": "initial_map", "source": source, "width": width, "height": int(width * min(aspect, 0.75)),
                "points": _between(rng, 2000, 20000 if source == "delaunay" else 400000)}
    width = _between(rng, 700, 3000)
    return {"kind": "pyramid", "width": width, "height": int(width * min(aspect, 2 / 3)), "levels": rng.randint(2, 3)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _cameras(count, width, height):
    """A reference pose 7 m from the scene, looking down at 45 degrees, and
    count - 1 poses on a ring of 0.8 m around it, all looking at the scene."""
    el = math.radians(45.0)
    K = syn.intrinsics(0.75 * width, width, height)
    centre = 7.0 * np.array([0.0, -math.cos(el), math.sin(el)])
    R0, T0 = syn.look_at(centre, np.zeros(3))
    cams = [(K, R0, T0)]
    for k in range(count - 1):
        a = 2 * math.pi * k / (count - 1)
        R, T = syn.look_at(centre + 0.8 * (math.cos(a) * R0[0] + math.sin(a) * R0[1]), np.zeros(3))
        cams.append((K, R, T))
    return cams


def _scene(count, width, height, seed):
    """(cameras, images, depth maps, normal maps): what the cameras see."""
    terrain = syn.ring_terrain(seed=seed)
    # The texture's finest detail stays at a few pixels whatever the image's size.
    terrain.texel = 0.06 * 1600.0 / width
    terrain.step = 0.05
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)
    cams = _cameras(count, width, height)
    images, depths, normals = [], [], []
    for K, R, T in cams:
        albedo, depth, normal = syn.render_aerial(terrain, K, R, T, width, height)
        grey = albedo * (255.0 * float(rng.uniform(0.8, 1.2)))
        grey = grey + 2.0 * torch.randn(grey.shape, generator=gen, device="cuda")
        images.append(torch.clamp(torch.round(grey), 0, 255))
        depths.append(depth)
        normals.append(normal)
    return cams, images, depths, normals, gen


def _estimated(depth, normal, gen):
    """The maps a PatchMatch pass leaves: relative depth noise, outliers, holes
    and perturbed normals."""
    r = torch.rand(depth.shape, generator=gen, device="cuda")
    d = depth * (1.0 + 0.002 * torch.randn(depth.shape, generator=gen, device="cuda"))
    wild = depth * (0.5 + torch.rand(depth.shape, generator=gen, device="cuda"))
    d = torch.where(r < 0.03, wild, torch.where(r < 0.05, torch.zeros_like(d), d))
    n = normal + math.radians(3.0) * torch.randn(normal.shape, generator=gen, device="cuda")
    n = n / torch.clamp(n.norm(dim=0, keepdim=True), min=1e-12)
    return d.contiguous(), n.contiguous()


def _range(depths):
    valid = depths[0][depths[0] > 0]
    return float(valid.min()) * 0.9, float(valid.max()) * 1.1


def _options(case, lo, hi, seed, mode, storage):
    photometric = mode == "photometric"
    return PatchMatchOptions(depth_min=lo, depth_max=hi, window_radius=case["radius"], window_step=case["step"],
                             sigma_spatial=case["radius"], num_iterations=case["iterations"],
                             geom_consistency=not photometric, init_depth_random=photometric,
                             image_storage=STORAGE[storage], random_seed=seed)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "stream": torch.cuda.Stream()}
    w, h = case["width"], case["height"]
    if kind == "depth_map":
        cams, images, depths, normals, gen = _scene(case["sources"] + 1, w, h, seed)
        geometric = case["mode"] == "geometric"
        views = []
        for (K, R, T), image, d, n in zip(cams, images, depths, normals):
            ed, en = _estimated(d, n, gen) if geometric else (None, None)
            views.append(View(image, K, R, T, depth=ed, normal=en))
        lo, hi = _range(depths)
        state["options"] = _options(case, lo, hi, seed, case["mode"], case["storage"])
        state["problem"] = Problem(0, list(range(1, len(views))), views)
    elif kind == "pool":
        # Every second view at full size, the others at two thirds of it.
        state["pool"] = pool = DepthMapPool(memory_budget_bytes=8 << 30, max_active_jobs=case["jobs"],
                                            image_storage=STORE_F16)
        state["jobs"], state["maps"] = [], []
        count = 8
        big = _scene(count, w, h, seed)
        small = _scene(count, w * 2 // 3, h * 2 // 3, seed)
        torch.cuda.synchronize()
        for k in range(count):
            cams, images = (big if k % 2 == 0 else small)[:2]
            pool.add_view(k, View(images[k], *cams[k]))
        lo, hi = _range(big[2])
        for j in range(case["jobs"]):
            ref = j % count
            sources = [(ref + 1 + i) % count for i in range(3 + j % 5)]
            state["jobs"].append((_options(case, lo, hi, seed + j, "photometric", "f16"), ref, sources))
            shape = big[1][ref].shape if ref % 2 == 0 else small[1][ref].shape
            state["maps"].append({name: torch.empty((3, *shape) if name == "normal" else tuple(shape), device="cuda")
                                  for name in ("depth", "normal", "conf")})
        torch.cuda.synchronize()
    elif kind == "cross_filter":
        cams, images, depths, normals, gen = _scene(case["views"], w, h, seed)
        maps = [_estimated(d, n, gen) for d, n in zip(depths, normals)]
        views = [View(None, *cam, depth=d, normal=n) for cam, (d, n) in zip(cams, maps)]
        ids = list(range(len(views)))
        state["problems"] = filter_problems(ids, [[s for s in ids if s != r] for r in ids], views)
        state["ids"] = ids
    elif kind == "fusion":
        cams, images, depths, normals, gen = _scene(case["views"], w, h, seed)
        state["images"], state["overlaps"] = [], []
        for (K, R, T), image, d, n in zip(cams, images, depths, normals):
            ed, en = _estimated(d, n, gen)
            grey = image.to(torch.int32)
            color = torch.stack([grey, (grey * 3 + 17) % 256, 255 - grey], -1).to(torch.uint8)
            state["images"].append(FusionImage(K=K, R=R, T=T, depth=ed, normal=en, color=color.contiguous()))
        centres = np.array([-R.T @ T for _, R, T in cams])
        for k in range(len(cams)):
            order = np.argsort(np.linalg.norm(centres - centres[k], axis=1), kind="stable")
            state["overlaps"].append([int(i) for i in order if i != k])
        # Where the program keeps the cloud: a point, its images and the end of their list.
        cap = len(cams) * w * h // 16
        state["cloud"] = {"points": np.zeros(cap, native.FUSED_POINT_DTYPE), "ends": np.zeros(cap, np.int64),
                          "seen_by": np.zeros(4 * cap, np.int32)}
    elif kind == "initial_map":
        cams, images, depths, normals, gen = _scene(1, w, h, seed)
        state["camera"] = K, R, T = cams[0]
        depth, normal = depths[0], normals[0]
        if case["source"] == "mesh":
            # The surface on a pixel grid, two triangles a cell, wound so that they face the camera.
            step = max(1, int(round(math.sqrt(w * h / max(case["points"], 1)))))
            ys, xs = torch.arange(0, h, step, device="cuda"), torch.arange(0, w, step, device="cuda")
            ny, nx = len(ys), len(xs)
            ys, xs = (g.reshape(-1) for g in torch.meshgrid(ys, xs, indexing="ij"))
            fy = fx = torch.zeros(len(ys), dtype=torch.float64, device="cuda")
        else:
            count = case["points"]
            ys = torch.randint(0, h, (count,), generator=gen, device="cuda")
            xs = torch.randint(0, w, (count,), generator=gen, device="cuda")
            fy = 0.2 + 0.6 * torch.rand(count, generator=gen, device="cuda", dtype=torch.float64)
            fx = 0.2 + 0.6 * torch.rand(count, generator=gen, device="cuda", dtype=torch.float64)
        d = depth[ys, xs].double()
        pixel = torch.stack([xs + fx, ys + fy, torch.ones_like(fx)], -1)
        cam_points = (pixel @ torch.tensor(np.linalg.inv(K).T, device="cuda")) * d[:, None]
        Rt = torch.tensor(R, device="cuda")
        points = (cam_points - torch.tensor(T, device="cuda")) @ Rt
        if case["source"] == "mesh":
            index = torch.arange(ny * nx, device="cuda").reshape(ny, nx)
            a, b = index[:-1, :-1].reshape(-1), index[:-1, 1:].reshape(-1)
            c, e = index[1:, :-1].reshape(-1), index[1:, 1:].reshape(-1)
            faces = torch.cat([torch.stack([a, c, b], 1), torch.stack([b, c, e], 1)])
            faces = faces[(d[faces] > 0).all(1)]
            p0, p1, p2 = (points[faces[:, k]] for k in range(3))
            n = torch.linalg.cross(p1 - p0, p2 - p0)
            n = n / torch.clamp(n.norm(dim=1, keepdim=True), min=1e-300)
            centre = torch.tensor(-R.T @ T, device="cuda")
            away = (((p0 + p1 + p2) / 3 - centre) * n).sum(1) > 0
            n[away] *= -1
            state["model"] = (points.contiguous(), faces.to(torch.int32).contiguous(), n.contiguous())
        else:
            seen = d > 0
            points = points * (1.0 + 1e-4 * torch.randn(points.shape, generator=gen, device="cuda",
                                                        dtype=torch.float64))
            state["model"] = (points[seen].float().contiguous(),
                              (normal[:, ys, xs].T.double() @ Rt)[seen].float().contiguous())
    else:
        cams, images, depths, normals, gen = _scene(1, w, h, seed)
        state["image"] = images[0]
        state["sizes"] = [pyramid.level_size(w, h, level)[:2] for level in range(case["levels"])]
        cw, ch = state["sizes"][-1]
        ys = (torch.arange(ch, device="cuda") * (h / ch)).long()
        xs = (torch.arange(cw, device="cuda") * (w / cw)).long()
        state["coarse"] = _estimated(depths[0][ys][:, xs], normals[0][:, ys][:, :, xs], gen)
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
class _Map:
    """A device map of the framework, for torch."""

    def __init__(self, pointer, shape, kind):
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": kind, "data": (int(pointer), False),
                                         "version": 3, "strides": None}


def _copy(pointer, shape, kind):
    return torch.as_tensor(_Map(pointer, shape, kind), device="cuda").clone()


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "depth_map":
        with PatchMatchACMMCuda(state["options"], state["problem"]) as pm:
            pm.Run()
            return {"depth": pm.GetDepthMap(), "normal": pm.GetNormalMap(), "conf": pm.GetConfMap()}
    if kind == "pool":
        pool = state["pool"]
        ids = [pool.submit(*job) for job in state["jobs"]]
        pool.run_until_done(ids)
        for job, maps in zip(ids, state["maps"]):
            pool.get_map(job, native.MAP_DEPTH, out=maps["depth"])
            pool.get_map(job, native.MAP_NORMAL, out=maps["normal"])
            pool.get_map(job, native.MAP_CONF, out=maps["conf"])
            pool.release(job)
        return state["maps"]
    if kind == "cross_filter":
        with torch.cuda.stream(state["stream"]):
            with CrossFilterCuda(PatchMatchOptions(), state["problems"], state["ids"], [True] * len(state["ids"]),
                                 stream=state["stream"].cuda_stream) as cf:
                cf.Run()
                cf.DedupRun()
                if case["host"]:
                    return [[cf.GetRefineDepthMap(k), cf.GetDeduplicDepthMap(k), cf.GetDeltDepthMap(k)]
                            for k in state["ids"]]
                out = []
                for k in state["ids"]:
                    maps = cf.DeviceMaps(k)
                    shape = (case["height"], case["width"])
                    out.append([_copy(maps["refined"], shape, "<f4"), _copy(maps["delta"], shape, "<f4"),
                                _copy(maps["visibility"], shape, "<i4")])
                return out
    if kind == "fusion":
        with StereoFusion(FusionOptions(), state["images"], state["overlaps"]) as fusion:
            fusion.Run()
            dropped = [fusion.RemoveDuplicatePoints(), fusion.RemoveOutliers()] if case["clean"] else []
            points = fusion.GetFusedPoints()
            offsets, seen_by = fusion.VisibilityCSR()
        cloud = state["cloud"]
        for name, part in (("points", points), ("ends", offsets[1:]), ("seen_by", seen_by)):
            cloud[name][:len(part)] = part
            cloud[name][len(part):] = 0
        points = cloud["points"]
        return {"dropped": dropped, "count": len(offsets) - 1, "ends": cloud["ends"], "seen_by": cloud["seen_by"],
                **{name: points[name] for name in ("x", "y", "z", "nx", "ny", "nz", "r", "g", "b", "score")}}
    if kind == "initial_map":
        build = {"sparse": init_maps.init_depth_from_sparse_points, "delaunay": init_maps.init_depth_from_delaunay,
                 "mesh": init_maps.init_depth_from_mesh, "dense": init_maps.init_depth_from_dense_points}
        model = state["model"][:1] if case["source"] in ("sparse", "delaunay") else state["model"]
        depth, normal, limits = build[case["source"]](case["width"], case["height"], *state["camera"], *model)
        return {"depth": depth, "normal": normal, "limits": list(limits)}
    stream = state["stream"]
    with torch.cuda.stream(stream):
        images = [pyramid.rescale_image(state["image"], w, h, stream.cuda_stream)[0]
                  for w, h in state["sizes"][1:]]
        maps = [state["coarse"]]
        for w, h in reversed(state["sizes"][:-1]):
            maps.append(pyramid.resample_maps(*maps[-1], w, h, stream.cuda_stream))
    return {"images": images, "maps": maps[1:]}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _window_flops(pixels, sources, case):
    """25 operations a window sample, 14 hypotheses a pixel and iteration, and
    5 more from the fourth iteration on."""
    taps = (2 * case["radius"] // case["step"] + 1) ** 2
    hypotheses = 14 * case["iterations"] + 5 * max(0, case["iterations"] - 3)
    return 25.0 * pixels * sources * taps * hypotheses


def work(case):
    kind = case["kind"]
    w, h = case["width"], case["height"]
    pixels = w * h
    if kind == "depth_map":
        n = case["sources"]
        read = 4 * (n + 1) + (4 * n + 16 if case["mode"] == "geometric" else 0)
        return {"bytes": pixels * (read + 20), "flops": _window_flops(pixels, n, case)}
    if kind == "pool":
        total = {"bytes": 0.0, "flops": 0.0}
        for j in range(case["jobs"]):
            p = pixels if j % 2 == 0 else (w * 2 // 3) * (h * 2 // 3)
            n = 3 + j % 5
            total["bytes"] += p * (2 * (n + 1) + 20)
            total["flops"] += _window_flops(p, n, case)
        return total
    if kind == "cross_filter":
        n = case["views"]
        return {"bytes": n * pixels * (16 + 12), "flops": 2 * 100.0 * n * (n - 1) * pixels}
    if kind == "fusion":
        # Maps and colours in, and about one point of 44 bytes and its images for every 50 pixels out.
        n = case["views"]
        return {"bytes": n * pixels * (19 + (44 + 4 * n) / 50), "flops": 40.0 * n * (n - 1) * pixels}
    if kind == "initial_map":
        per = {"sparse": 12, "delaunay": 12, "dense": 24, "mesh": 72}[case["source"]]
        return {"bytes": pixels * 16 + per * case["points"], "flops": 0}
    sizes = [pyramid.level_size(w, h, level)[:2] for level in range(case["levels"])]
    areas = [a * b for a, b in sizes]
    return {"bytes": 4 * (areas[0] + sum(areas[1:])) + 16 * (areas[-1] + sum(areas[:-1])), "flops": 0}


# ---------------------------------------------------------------------------
# In 64 bits
# ---------------------------------------------------------------------------
def _filter(n, out):
    """The (out, n) matrix of the triangle filter, widened when minifying."""
    scale = out / n
    wide = min(scale, 1.0)
    centre = (torch.arange(out, dtype=torch.float64, device="cuda") + 0.5) / scale
    place = torch.arange(n, dtype=torch.float64, device="cuda") + 0.5
    weight = torch.clamp(1.0 - (place[None] - centre[:, None]).abs() * wide, min=0.0)
    return weight / weight.sum(1, keepdim=True)


def _bilinear(maps, w, h):
    """Bilinear samples of (planes, rows, cols) at the centres of a w x h grid, zero outside."""
    planes, rows, cols = maps.shape
    padded = torch.nn.functional.pad(maps, (1, 1, 1, 1))
    r = (torch.arange(h, dtype=torch.float64, device="cuda") + 0.5) * (rows / h) - 0.5
    c = (torch.arange(w, dtype=torch.float64, device="cuda") + 0.5) * (cols / w) - 0.5
    r0, c0 = torch.floor(r), torch.floor(c)
    fr, fc = (r - r0)[:, None], (c - c0)[None, :]
    r0, c0 = r0.long() + 1, c0.long() + 1

    def at(y, x):
        return padded[:, y][:, :, x]
    top = (1 - fc) * at(r0, c0) + fc * at(r0, c0 + 1)
    low = (1 - fc) * at(r0 + 1, c0) + fc * at(r0 + 1, c0 + 1)
    return (1 - fr) * top + fr * low


def exact(case, seed):
    """The pyramid's outputs. The other paths choose between random or
    neighbouring hypotheses, or accept and reject by thresholds, step after
    step: there is no value in 64 bits that they approach."""
    if case["kind"] != "pyramid":
        return None
    state = prepare(case, seed)
    image = state["image"].double()
    images = []
    for w, h in state["sizes"][1:]:
        out = _filter(case["height"], h) @ (image @ _filter(case["width"], w).T)
        images.append(torch.clamp(torch.round(out), 0, 255))
    depth, normal = (m.double() for m in state["coarse"])
    maps = []
    for w, h in reversed(state["sizes"][:-1]):
        depth = _bilinear(depth[None], w, h)[0]
        normal = _bilinear(normal, w, h)
        size = normal.square().sum(0, keepdim=True).sqrt()
        normal = torch.where(size > 0, normal / torch.where(size > 0, size, torch.ones_like(size)), normal)
        maps.append((depth, normal))
    return {"images": images, "maps": maps}
