"""Performance cases: the work a program gives this renderer, through its public Python API.

listed() names the cases, draw(rng) makes more of the same ranges, prepare() builds
what a program holds before the call (a scene resident on the GPU, accumulators,
rays), run() makes one call and returns what it produced, exact() gives the
outputs that have a value in 64-bit arithmetic, and work() the bytes and
operations one call cannot do without.

Every kind of case is one entry point:
    frame      render_device: a stream-ordered render into device accumulators
    host       render_image: a render into a host PixelBuffer, copies included
    batch      render_batch: jobs of several scenes and sizes in one call
    served     Server: a burst of requests with their own cameras, stepped until done
    closest    Scene.intersect: closest hits of host rays
    occluded   Scene.occluded: any hit of host rays
    film       resolve_srgb: accumulators to sRGB bytes
"""

from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

import albedo_b200 as ab
from albedo_b200 import scenes

METHODS = {"megakernel": ab.MEGAKERNEL, "wavefront": ab.WAVEFRONT}
ESTIMATORS = {"path": ab.PATH, "scatter": ab.SCATTER_ONLY, "normals": ab.NORMALS}
SUMS = {"fp64": ab.ACCUMULATE_FP64, "kahan": ab.ACCUMULATE_KAHAN_FP32}

EYE, TARGET, UP, FOV = (0.0, 2.4, 7.8), (0.0, 1.9, -0.5), (0.0, 1.0, 0.0), 38.0


def _frame(name, scene, width, height, n, depth, **more):
    case = {"name": name, "kind": "frame", "scene": scene, "detail": 0, "smooth": True, "width": width,
            "height": height, "n": n, "depth": depth, "method": "megakernel", "estimator": "path", "sums": "fp64"}
    return {**case, **more}


def listed():
    return [
        # A material or thumbnail preview: one sample a pixel, nothing but latency.
        _frame("thumbnail", "room", 64, 36, 1, 8),
        # The plain configuration as a drop-in caller makes it: the analytic-sphere
        # room at 320x180, 16 samples, into a host PixelBuffer.
        _frame("room_host", "room", 320, 180, 4, 8, kind="host"),
        # The instanced-mesh configuration: three smooth trefoil tubes (16,384
        # triangles) in gold, glass and copper, 960x540, 64 samples.
        _frame("knots_frame", "knots", 960, 540, 8, 10, detail=256),
        # The large-mesh configuration: a displaced icosphere of 1.31M triangles in
        # rough glass at 1920x1080, with the samples of an interactive final.
        _frame("ball_frame", "ball", 1920, 1080, 6, 16, detail=8),
        # The random-triangle stress scene with compensated FP32 sums, ragged size.
        _frame("soup_kahan", "soup", 853, 481, 4, 12, detail=200_003, smooth=False, sums="kahan"),
        # A normals pass, as written beside a render for a denoiser: one sample, odd size.
        _frame("normals_pass", "knots", 641, 361, 1, 1, detail=128, smooth=False, estimator="normals"),
        # The wavefront form of one frame.
        _frame("wavefront_frame", "knots", 960, 540, 4, 10, detail=256, method="wavefront"),
        # A farm's batch: uneven jobs over several scenes in one call.
        {"name": "batch", "kind": "batch", "scenes": 6, "jobs": 16, "depth": 16},
        # A render server taking a burst of small and large requests.
        {"name": "served", "kind": "served", "scenes": 4, "jobs": 12, "depth": 12},
        # Ray queries from a simulation: hits with their geometry.
        {"name": "closest", "kind": "closest", "scene": "knots", "detail": 128, "smooth": False, "count": 1 << 18,
         "geometry": True},
        # Visibility between points, a ragged million of them.
        {"name": "occluded", "kind": "occluded", "scene": "knots", "detail": 256, "smooth": False,
         "count": 1_000_003},
        # A 4K film written as sRGB bytes.
        {"name": "film_4k", "kind": "film", "width": 3840, "height": 2160},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng: random.Random):
    kind = rng.choice(["frame", "frame", "frame", "host", "batch", "served", "closest", "occluded", "film"])
    if kind in ("batch", "served"):
        return {"kind": kind, "scenes": rng.randint(1, 6), "jobs": rng.randint(2, 16), "depth": rng.randint(4, 16)}
    if kind == "film":
        return {"kind": kind, "width": _log_int(rng, 16, 3840), "height": _log_int(rng, 16, 2160)}
    scene = rng.choice(["room", "knots", "ball", "soup"])
    detail = {"room": 0, "knots": 8 * _log_int(rng, 4, 32), "ball": rng.randint(2, 6),
              "soup": _log_int(rng, 1000, 300_000)}[scene]
    if kind in ("closest", "occluded"):
        case = {"kind": kind, "scene": scene, "detail": detail, "smooth": False, "count": _log_int(rng, 100, 1 << 20)}
        return {**case, "geometry": rng.random() < 0.5} if kind == "closest" else case
    width = _log_int(rng, 32, 1920)
    height = max(8, int(width * rng.uniform(0.5, 0.8)))
    n = min(rng.randint(1, 8), max(1, int(math.sqrt(2.0e7 / (width * height)))))
    case = _frame("", scene, width, height, n, rng.randint(2, 16), detail=detail, kind=kind,
                  smooth=scene != "soup" and rng.random() < 0.7)
    option = rng.choice(["plain", "plain", "wavefront", "kahan", "scatter", "normals"])
    if option == "wavefront":
        case["method"] = "wavefront"
    elif option == "kahan":
        case["sums"] = "kahan"
    elif option != "plain":
        case["estimator"] = option
    del case["name"]
    return case


# ---------------------------------------------------------------- scenes


def _materials(scene):
    conductor = functools.partial(ab.BasicMaterial, "conductor")
    glass = functools.partial(ab.BasicMaterial, "dielectric", ior=1.5)
    basic = {
        "gold": conductor(a=(0.156, 0.424, 1.383), b=(3.602, 2.472, 1.915), roughness=0.25),
        "silver": conductor(a=(0.155, 0.117, 0.138), b=(4.83, 3.12, 2.15)),
        "copper": conductor(a=(0.238, 1.007, 1.240), b=(3.626, 2.582, 2.393), roughness=0.3),
        "glass": glass(),
        "rough_glass": glass(roughness=0.447),
        "frosted": glass(roughness=0.316),
        "white": ab.BasicMaterial(a=(0.73, 0.73, 0.73)),
        "red": ab.BasicMaterial(a=(0.63, 0.07, 0.05)),
        "green": ab.BasicMaterial(a=(0.12, 0.45, 0.15)),
        "blue": ab.BasicMaterial(a=(0.15, 0.3, 0.7)),
        "tiles": ab.BasicMaterial(texture="checker", a=(0.73, 0.73, 0.73), b=(0.3, 0.3, 0.3),
                                  frequency_or_scale=1.25),
    }
    index = {name: scene.add_material(m) for name, m in basic.items()}
    index["mixed"] = scene.add_material(basic["gold"], basic["white"], scale=2.0, veins=6.0, threshold=0.5)
    return index


def _floor():
    points = np.array([[-3.5, 0, 12], [3.5, 0, 12], [3.5, 0, -4.5], [-3.5, 0, -4.5]], np.float64)
    return points, np.array([[0, 1, 2], [0, 2, 3]])


@functools.lru_cache(maxsize=8)
def _sphere_points(level):
    return scenes.icosphere(level)


def _ball(level, rng):
    """An icosphere displaced by a few seeded plane waves."""
    points, faces = _sphere_points(level)
    waves = rng.normal(size=(6, 3)) * np.array([2, 2, 4, 4, 8, 8])[:, None]
    height = sum(np.sin(points @ w + p) / np.linalg.norm(w) for w, p in zip(waves, rng.uniform(0, 6.28, 6)))
    return (points * (1.0 + 0.08 * height)[:, None]).astype(np.float32), faces


def _knot(segments):
    points, quads = scenes.trefoil_mesh(segments, segments // 8)
    return points, np.concatenate([quads[:, [0, 1, 2]], quads[:, [0, 2, 3]]])


def _soup(count, rng):
    centers = rng.uniform(-0.5, 0.5, size=(count, 1, 3))
    lengths = np.exp(rng.uniform(math.log(1e-3), math.log(3e-2), size=(count, 1, 1)))
    corners = rng.normal(size=(count, 3, 3)) * lengths
    return (centers + corners).reshape(-1, 3).astype(np.float32), np.arange(3 * count).reshape(-1, 3)


def _placement(points, size, angle, position):
    """Scales the points' longest extent to `size`, turns them about y and stands them at `position`."""
    low, high = points.min(axis=0).astype(np.float64), points.max(axis=0).astype(np.float64)
    scale = size / (high - low).max()
    c, s = math.cos(angle), math.sin(angle)
    linear = scale * np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]])
    middle = np.array([(low[0] + high[0]) / 2, low[1], (low[2] + high[2]) / 2])
    offset = np.array(position) - linear @ middle
    inverse = np.linalg.inv(linear)
    return np.column_stack([linear, offset]), np.column_stack([inverse, -inverse @ offset])


def _parts(kind, detail, seed, look="frosted"):
    """The seeded scene as plain data: spheres (centre, radius, material), meshes (points, faces) and
    instances (mesh, to_world, to_object, material)."""
    rng = np.random.default_rng([seed, detail])
    spheres, meshes, instances = [], [], []
    if kind in ("room", "knots"):
        spheres += [((0, 0, -10004), 10000, "white"), ((-10003, 0, 0), 10000, "red"),
                    ((10003, 0, 0), 10000, "green")]
        spheres.append(((0, -10000 if kind == "room" else 10005, 0), 10000, "white"))
    if kind == "room":
        for x, z, m in [(-2.2, -1.2, "glass"), (-1.1, 0.6, "rough_glass"), (0.0, -1.6, "silver"),
                        (1.1, 0.6, "gold"), (2.2, -1.2, "blue")]:
            dx, dz = rng.uniform(-0.1, 0.1, 2)
            spheres.append(((x + dx, 0.8, z + dz), 0.8, m))
        return spheres, meshes, instances
    meshes.append(_floor())
    still = np.eye(3, 4)
    instances.append((0, still, still, "tiles"))
    if kind == "knots":
        meshes.append(_knot(detail))
        for m, x, z in [("gold", -1.7, -1.4), ("glass", 0.0, 0.4), ("copper", 1.7, -1.4)]:
            instances.append((1, *_placement(meshes[1][0], 1.6 * rng.uniform(0.8, 1.2), rng.uniform(0, 6.28),
                                             (x, 0, z)), m))
    elif kind == "ball":
        meshes.append(_ball(detail, rng))
        instances.append((1, *_placement(meshes[1][0], 2.6, rng.uniform(0, 6.28), (0, 0, -0.5)), look))
    else:
        meshes.append(_soup(detail, rng))
        instances.append((1, *_placement(meshes[1][0], 3.0, rng.uniform(0, 6.28), (0, 0, -0.5)), "gold"))
    return spheres, meshes, instances


def _resident(parts, camera, smooth, lights=True):
    spheres, meshes, instances = parts
    scene = ab.Scene.create()
    scene.set_camera(*camera)
    material = _materials(scene)
    for i, (points, faces) in enumerate(meshes):
        if i == 0:  # the floor, textured by its own x and z
            scene.add_mesh(points, faces, uvs=points[:, [0, 2]], texture_faces=faces)
        else:
            scene.add_mesh(points, faces, smooth=smooth)
    for centre, radius, m in spheres:
        scene.add_sphere(centre, radius, material[m])
    for mesh, to_world, to_object, m in instances:
        scene.add_instance(mesh, to_world, to_object, material[m])
    if lights:
        scene.add_area_light((0, 5.6, -1.2), 1.1, (9, 7.6, 5.8), material["white"])
        scene.add_point_light((0.8, 4.2, 3.2), (1.2, 2.0, 3.6))
        scene.set_sky((0.05, 0.06, 0.08))
    scene.commit()
    return scene


def _view(seed):
    """A seeded camera near the scenes' usual one."""
    rng = np.random.default_rng([seed, 1])
    eye = tuple(float(v) for v in np.array(EYE) + rng.uniform(-0.4, 0.4, 3))
    return eye, TARGET, UP, FOV


def _rays(count, seed):
    """Rays between points around the objects, as a simulation draws them: origins in the volume
    above the floor, unit directions over the sphere."""
    rng = np.random.default_rng([seed, 2])
    origins = rng.uniform([-3.0, 0.05, -3.5], [3.0, 4.0, 4.0], size=(count, 3))
    directions = rng.normal(size=(count, 3))
    directions /= np.linalg.norm(directions, axis=1, keepdims=True)
    return np.concatenate([origins, directions], axis=1).astype(np.float32)


# ---------------------------------------------------------------- preparing and running


def _accumulators(width, height):
    return torch.zeros((width * height, 4), dtype=torch.float64, device="cuda")


def _film(acc):
    """The accumulators as the renderer fills them: FP64 sums and, in the fourth field, int64 counts."""
    return {"sums": acc[:, :3], "count": acc.view(torch.int64)[:, 3]}


def _job(case, seed):
    return ab.RenderJob(case["width"], case["height"], samples_per_axis=case["n"], seed=seed,
                        estimator=ESTIMATORS[case["estimator"]], max_depth=case["depth"],
                        method=METHODS[case["method"]], accumulation=SUMS[case["sums"]])


def _mixed_jobs(case, seed):
    """Scenes and jobs of uneven size: displaced icospheres of 320 to 82k triangles with some spheres
    around them, image sizes and samples over their ranges. Sizes depend on the case alone."""
    sizes = random.Random(case["scenes"] * 1000 + case["jobs"])
    stages = []
    for s in range(case["scenes"]):
        look = ["frosted", "gold", "white", "mixed"][s % 4]
        spheres, meshes, instances = _parts("ball", sizes.randint(2, 6), seed * 64 + s, look)
        rng = np.random.default_rng([seed, s, 3])
        for _ in range(sizes.randint(0, 8)):
            r = float(rng.uniform(0.2, 0.5))
            spheres.append(((float(rng.uniform(-2.5, 2.5)), r, float(rng.uniform(-2.5, 1.5))), r,
                            ["white", "gold", "frosted", "mixed"][rng.integers(4)]))
        stages.append(_resident((spheres, meshes, instances), (EYE, TARGET, UP, FOV), True))
    jobs = []
    for j in range(case["jobs"]):
        width, height = sizes.choice(scenes.RESOLUTIONS)
        jobs.append((stages[j % len(stages)], ab.RenderJob(width, height, samples_per_axis=sizes.randint(2, 6),
                                                           seed=seed + j, max_depth=case["depth"]),
                     _accumulators(width, height), ab.Camera(*_view(seed * 64 + j))))
    return stages, jobs


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "served"):
        stages, jobs = _mixed_jobs(case, seed)
        state = {"kind": kind, "stages": stages, "jobs": jobs}
        if kind == "served":
            state["server"] = ab.Server()
        return state
    if kind == "film":
        generator = torch.Generator(device="cuda").manual_seed(seed)
        pixels = case["width"] * case["height"]
        acc = _accumulators(case["width"], case["height"])
        # Averages from black to a few times white, as a rendered frame has, at 36 or 64 samples a pixel.
        counts = torch.where(torch.rand(pixels, generator=generator, device="cuda") < 0.5, 36, 64)
        level = torch.randn((pixels, 3), generator=generator, device="cuda", dtype=torch.float64)
        acc[:, :3] = torch.exp(1.5 * level - 1.5) * counts[:, None]
        acc.view(torch.int64)[:, 3] = counts
        out = torch.empty(3 * pixels, dtype=torch.uint8, device="cuda")
        return {"kind": kind, "width": case["width"], "height": case["height"], "acc": acc, "out": out}
    scene = _resident(_parts(case["scene"], case["detail"], seed), _view(seed), case["smooth"])
    if kind in ("closest", "occluded"):
        state = {"kind": kind, "scene": scene, "rays": _rays(case["count"], seed)}
        if kind == "closest":
            state["geometry"] = case["geometry"]
        else:
            state["range"] = np.random.default_rng([seed, 4]).uniform(0.5, 6.0, case["count"]).astype(np.float32)
        return state
    state = {"kind": kind, "scene": scene, "job": _job(case, seed)}
    if kind == "host":
        state["image"] = ab.PixelBuffer(case["width"], case["height"])
    else:
        state["acc"] = _accumulators(case["width"], case["height"])
    return state


def run(state):
    kind = state["kind"]
    if kind == "frame":
        ab.render_device(state["scene"], state["job"], state["acc"].data_ptr())
        return _film(state["acc"])
    if kind == "host":
        ab.render_image(state["scene"], state["job"], state["image"])
        pixels = state["image"].pixels
        return {"sums": pixels.view(np.float64).reshape(-1, 4)[:, :3], "count": pixels["count"]}
    if kind == "batch":
        ab.render_batch([(scene, job, acc.data_ptr()) for scene, job, acc, _ in state["jobs"]])
        return [_film(acc) for _, _, acc, _ in state["jobs"]]
    if kind == "served":
        server = state["server"]
        waiting = {server.submit(scene, job, acc.data_ptr(), camera) for scene, job, acc, camera in state["jobs"]}
        while waiting:
            waiting.difference_update(server.step())
        return [_film(acc) for _, _, acc, _ in state["jobs"]]
    if kind == "closest":
        return state["scene"].intersect(state["rays"], geometry=state["geometry"])
    if kind == "occluded":
        return state["scene"].occluded(state["rays"], state["range"])
    ab.resolve_srgb(state["acc"].data_ptr(), state["width"], state["height"], state["out"].data_ptr())
    return state["out"]


# ---------------------------------------------------------------- 64-bit values


def _world_triangles(parts):
    _, meshes, instances = parts
    corners = []
    for mesh, to_world, _, _ in instances:
        points, faces = meshes[mesh]
        world = points.astype(np.float64) @ to_world[:, :3].T + to_world[:, 3]
        corners.append(world[np.asarray(faces)])
    return np.concatenate(corners) if corners else np.zeros((0, 3, 3))


def _nearest(parts, lights, origins, directions):
    """Closest hits of FP64 rays by testing every primitive: distance (inf: none) and outward unit normal."""
    device = "cuda" if torch.cuda.is_available() else "cpu"
    o = torch.from_numpy(origins).to(device)
    d = torch.from_numpy(directions).to(device)
    tri = torch.from_numpy(_world_triangles(parts)).to(device)
    best = torch.full((len(o),), math.inf, dtype=torch.float64, device=device)
    normal = torch.zeros_like(o)
    for centre, radius in [(c, r) for c, r, _ in parts[0]] + lights:
        oc = o - torch.tensor(centre, dtype=torch.float64, device=device)
        a, h = (d * d).sum(1), (d * oc).sum(1)
        c = (oc * oc).sum(1) - radius * radius
        disc = h * h - a * c
        q = -(h + torch.copysign(torch.sqrt(disc.clamp_min(0)), h))
        roots = torch.stack([q / a, c / q]).sort(dim=0).values
        for t in roots:
            nearer = (disc >= 0) & (t > 0) & (t < best)
            best = torch.where(nearer, t, best)
            normal = torch.where(nearer[:, None], (oc + d * t[:, None]) / radius, normal)
    if len(tri):
        v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
        face = torch.linalg.cross(e1, e2)
        unit = face / face.norm(dim=1, keepdim=True)
        # Moeller and Trumbore's test as matrix products: det = -d.n, t = (o - v0).n / det,
        # u = ((o x d).e2 - d.(e2 x v0)) / det, v = (d.(e1 x v0) - (o x d).e1) / det.
        moment = torch.linalg.cross(o, d)
        c1, c2, at = torch.linalg.cross(e1, v0), torch.linalg.cross(e2, v0), (v0 * face).sum(1)
        step = max(1, (1 << 26) // len(tri))
        for i in range(0, len(o), step):
            s = slice(i, i + step)
            det = -(d[s] @ face.T)
            t = (o[s] @ face.T - at) / det
            u = (moment[s] @ e2.T - d[s] @ c2.T) / det
            v = (d[s] @ c1.T - moment[s] @ e1.T) / det
            t = torch.where((u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0), t, math.inf)
            nearest, index = t.min(dim=1)
            nearer = nearest < best[s]
            best[s] = torch.where(nearer, nearest, best[s])
            normal[s] = torch.where(nearer[:, None], unit[index], normal[s])
    return best.cpu().numpy(), normal.cpu().numpy()


LIGHT = [((0, 5.6, -1.2), 1.1)]


def _exact_normals(case, seed):
    """The normals estimator in 64 bits: each pixel's own PCG32 stream jitters its samples; a hit gives
    0.5 (n + 1), a miss the gradient from white to (0.5, 0.7, 1)."""
    width, height, n = case["width"], case["height"], case["n"]
    y, x = np.divmod(np.arange(width * height, dtype=np.uint64), np.uint64(width))
    with np.errstate(over="ignore"):
        v = np.arange(width * height, dtype=np.uint64)
        v = (v ^ (v >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        v = (v ^ (v >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        inc = ((v ^ (v >> np.uint64(31))) << np.uint64(1)) | np.uint64(1)
        multiplier = np.uint64(6364136223846793005)
        state = (inc + np.uint64(seed)) * multiplier + inc

        def uniform():
            nonlocal state
            old = state
            state = old * multiplier + inc
            word = (((old >> np.uint64(18)) ^ old) >> np.uint64(27)).astype(np.uint32)
            turn = (old >> np.uint64(59)).astype(np.uint32)
            return ((word >> turn) | (word << ((np.uint32(32) - turn) & np.uint32(31)))) / 4294967296.0

        eye, target, up, fov = (np.array(v, np.float64) for v in _view(seed))
        back = (eye - target) / np.linalg.norm(eye - target)
        right = np.cross(up, back)
        right /= np.linalg.norm(right)
        half = math.tan(math.radians(float(fov)) / 2)
        total = np.zeros((width * height, 3))
        parts = _parts(case["scene"], case["detail"], seed)
        for sample in range(n * n):
            fx = (x + (sample % n + uniform()) / n) / width
            fy = (y + (sample // n + uniform()) / n) / height
            d = (-back + np.outer(2 * fx - 1, right * half * width / height)
                 + np.outer(1 - 2 * fy, np.cross(back, right) * half))
            d /= np.linalg.norm(d, axis=1, keepdims=True)
            t, normal = _nearest(parts, LIGHT, np.broadcast_to(eye, d.shape).copy(), d)
            normal = np.where(((normal * d).sum(1) > 0)[:, None], -normal, normal)
            h = 0.5 * (d[:, 1:2] + 1)
            total += np.where(np.isfinite(t)[:, None], 0.5 * (normal + 1), (1 - h) + h * np.array([0.5, 0.7, 1.0]))
    return {"sums": total, "count": None}


def exact(case, seed):
    """Path-traced images have no such value: each is a sum over random paths whose branches are taken by
    comparing FP32 numbers, and the renderer's are FP32 paths. Bytes, counts and ids are whole numbers."""
    kind = case["kind"]
    if case.get("smooth", True) or kind not in ("frame", "host", "closest"):
        return None
    triangles = {"room": 0, "knots": 3 * case["detail"] ** 2 // 4, "ball": 20 << (2 * case["detail"]),
                 "soup": case["detail"]}[case["scene"]]
    rays = case["count"] if kind == "closest" else case["width"] * case["height"] * case["n"] ** 2
    if rays * triangles > 4.0e9 or (kind != "closest" and case["estimator"] != "normals"):
        return None
    if kind != "closest":
        return _exact_normals(case, seed)
    rays = _rays(case["count"], seed).astype(np.float64)
    t, normal = _nearest(_parts(case["scene"], case["detail"], seed), LIGHT, rays[:, :3].copy(), rays[:, 3:].copy())
    hit = np.isfinite(t)
    out = {"hit": None, "object": None, "triangle": None, "t": np.where(hit, t, 0.0)}
    if case["geometry"]:
        facing = np.where(((normal * rays[:, 3:]).sum(1) > 0)[:, None], -normal, normal) * hit[:, None]
        out |= {"front": None, "normal": facing, "shading_normal": facing,
                "point": np.where(hit[:, None], rays[:, :3] + np.where(hit, t, 0.0)[:, None] * rays[:, 3:], 0.0)}
    return out


# ---------------------------------------------------------------- work


def _scene_bytes(kind, detail):
    """Geometry a query or render reads at least once: 36 bytes of positions a triangle and a 24-byte box for
    each of about half as many leaves."""
    triangles = {"room": 0, "knots": detail ** 2 // 4, "ball": 20 << (2 * detail), "soup": detail}[kind]
    return 48 * triangles + 1024


def _path_flops(kind, paths, depth, estimator="path"):
    """Roughly what a path costs: queries a path (closest-hit and shadow), 20 boxes a query at 15 operations
    and one primitive at 60, and 150 operations of shading a bounce."""
    queries = 1 if estimator == "normals" else min(2 * depth, {"room": 6, "knots": 7, "ball": 2, "soup": 4}[kind])
    return paths * queries * (20 * 15 + 60 + 75)


def work(case):
    kind = case["kind"]
    if kind in ("batch", "served"):
        sizes = random.Random(case["scenes"] * 1000 + case["jobs"])
        total = {"bytes": 0, "flops": 0}
        for _ in range(case["scenes"]):
            total["bytes"] += _scene_bytes("ball", sizes.randint(2, 6))
            sizes.randint(0, 8)
        for _ in range(case["jobs"]):
            width, height = sizes.choice(scenes.RESOLUTIONS)
            total["bytes"] += 64 * width * height
            total["flops"] += _path_flops("ball", width * height * sizes.randint(2, 6) ** 2, case["depth"])
        return total
    if kind == "film":
        pixels = case["width"] * case["height"]
        return {"bytes": 35 * pixels, "flops": 6 * pixels}
    geometry = _scene_bytes(case["scene"], case["detail"])
    if kind in ("closest", "occluded"):
        # A ray is 24 bytes; occluded adds its range and answer, closest its 16 or 56 bytes of outputs.
        per_ray = 32 if kind == "occluded" else 80 if case["geometry"] else 40
        return {"bytes": geometry + per_ray * case["count"], "flops": 360 * case["count"]}
    pixels = case["width"] * case["height"]
    return {"bytes": geometry + 64 * pixels,
            "flops": _path_flops(case["scene"], pixels * case["n"] ** 2, case["depth"], case["estimator"])}
