"""Performance cases of the path tracer: the calls that programs make through its public API.

Every case is one call a user waits for, from host inputs to host results: frames (`render`),
progressive sessions, batches of small jobs, building a scene and rendering it once, ray queries
and explicit paths. Scenes are the package's own seeded generators (the Cornell box, rooms filled
with displaced spheres, sphere fields, the same with a medium, with textures or with two levels);
the seed of a case moves the geometry, the rays and the random streams.

Images come back with the path counts of their statistics. The counts of box and triangle tests
are left out: they say how much work the traversal did, not what it computed.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from minirender_b200 import api, scene

MODES = ("mis", "light", "bsdf")


def listed():
    return [
        # A preview-sized frame of a trivial scene: nothing but launches and latency (material
        # previews, thumbnails, the first frame while a user drags the camera).
        {"name": "thumbnail", "call": "render", "scene": "cornell", "triangles": 36, "width": 64,
         "height": 64, "spp": 4, "depth": 8, "mode": "mis"},
        # The small benchmark frame: a trivial scene at an ordinary size, shading-heavy.
        {"name": "cornell_512", "call": "render", "scene": "cornell", "triangles": 36, "width": 512,
         "height": 512, "spp": 16, "depth": 8, "mode": "mis"},
        # An ordinary job of the uneven mix: odd square size, many materials, split references.
        {"name": "room_556", "call": "render", "scene": "room", "triangles": 261_000, "width": 556,
         "height": 556, "spp": 49, "depth": 11, "mode": "mis"},
        # The large frame: a million triangles, full HD, thin lens, environment and sun.
        {"name": "field_1080p", "call": "render", "scene": "field", "triangles": 1_024_000,
         "width": 1920, "height": 1080, "spp": 64, "depth": 12, "mode": "mis"},
        # A scene in a homogeneous medium: free flights, phase functions, long scattered paths.
        {"name": "fog_quarter_hd", "call": "render", "scene": "fog", "triangles": 1_024_000,
         "width": 961, "height": 541, "spp": 8, "depth": 16, "mode": "mis"},
        # Instances over per-mesh trees with textures, normal maps and an environment map.
        {"name": "instanced_textured", "call": "render", "scene": "instanced", "triangles": 512_000,
         "width": 641, "height": 359, "spp": 16, "depth": 8, "mode": "mis"},
        # An interactive session: the frame arrives in four committed batches of samples.
        {"name": "session", "call": "session", "scene": "room", "triangles": 60_000, "width": 400,
         "height": 300, "spp": 16, "depth": 8, "mode": "mis"},
        # Preview-sized jobs of a request queue, uneven scenes and depths, rendered together.
        {"name": "batch_previews", "call": "batch", "scene": "room", "triangles": 40_000, "jobs": 24,
         "width": 128, "height": 128, "spp": 4, "depth": 12, "mode": "mis"},
        # A one-shot command: upload the scene, build its tree, render one image, free it.
        {"name": "build_and_render", "call": "build", "scene": "room", "triangles": 480_000,
         "width": 256, "height": 256, "spp": 4, "depth": 6, "mode": "mis"},
        # Baking and simulation: nearest hits of many unordered rays.
        {"name": "nearest_hits", "call": "nearest", "scene": "room", "triangles": 30_000,
         "rays": 1_000_003},
        # Picking and visibility of a few points at a time: latency of a small query.
        {"name": "occlusion_small", "call": "occluded", "scene": "room", "triangles": 120_000,
         "rays": 1_021},
        # Radiance along explicit rays (light probes): a small wave of paths.
        {"name": "probe_paths", "call": "paths", "scene": "cornell", "triangles": 36, "rays": 4_099,
         "depth": 8, "mode": "mis"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(("render", "render", "render", "session", "batch", "build", "nearest",
                       "occluded", "paths"))
    kind = rng.choice(("cornell", "room", "field", "fog", "instanced"))
    if call in ("nearest", "occluded"):
        return {"call": call, "scene": "room", "triangles": _log_uniform(rng, 2_000, 500_000),
                "rays": _log_uniform(rng, 1, 1_500_000)}
    case = {"call": call, "scene": kind}
    case["triangles"] = 36 if kind == "cornell" else _log_uniform(
        rng, 10_000, 500_000 if kind == "room" else 1_000_000)
    case["depth"] = rng.randint(4, 12)
    case["mode"] = rng.choice(("mis", "mis", "mis", "light", "bsdf"))
    if call == "paths":
        case["rays"] = _log_uniform(rng, 1, 200_000)
        return case
    if call == "batch":
        case["jobs"] = _log_uniform(rng, 2, 40)
        case["width"] = case["height"] = _log_uniform(rng, 64, 256)
        case["spp"] = _log_uniform(rng, 1, 8)
        return case
    case["width"] = _log_uniform(rng, 48, 1024)
    case["height"] = max(32, round(case["width"] * rng.uniform(0.5, 1.0)))
    case["spp"] = _log_uniform(rng, 1, 32 if call == "render" else 8)
    return case


# ---- inputs ----

def _textured(document, rng):
    """Base-colour and normal textures on the document's materials and an environment map."""
    def smooth(height, width):
        coarse = rng.random((max(2, height // 8), max(2, width // 8), 3), dtype=np.float32)
        return np.repeat(np.repeat(coarse, 8, 0), 8, 1)[:height, :width]

    normals = np.full((128, 128, 3), (0.5, 0.5, 1.0), np.float32)
    normals[..., :2] += 0.2 * (smooth(128, 128)[..., :2] - 0.5)
    document.textures = [scene.TextureData(smooth(256, 256)), scene.TextureData(normals),
                         scene.TextureData(2.0 * smooth(128, 256))]
    for i, m in enumerate(document.materials):
        if m.kind == "diffuse":
            m.base_color_texture = 0
            if i % 2:
                m.normal_texture = 1
                m.normal_scale = 0.5
    document.environment_texture = 2
    # Spheres and ground get texture coordinates from their positions.
    for mesh in document.meshes:
        p = mesh.positions[mesh.corner_positions]
        mesh.corner_uvs = np.ascontiguousarray(p[..., :2] * np.float32(0.5) + np.float32(0.5))


def _document(kind, triangles, seed):
    if kind == "cornell":
        return scene.cornell_box()
    if kind == "room":
        return scene.job_scene(triangles, 1 + seed)
    spheres = max(1, triangles // 5120)
    document = scene.sphere_field(spheres, 20.0, 1 + seed % 10_000, subdivisions=4,
                                  variants=min(8, spheres))
    if kind == "fog":
        document.media = [scene.MediumRegion((-11.0, -1.0, -11.0), (11.0, 21.0, 11.0),
                                             (0.01, 0.02, 0.03), (0.1, 0.1, 0.1), 0.0)]
    if kind == "instanced":
        _textured(document, np.random.default_rng(seed))
    return document


def _build(kind, document):
    """The scene on the GPU with the builder options its kind is used with."""
    return api.Scene(document, split_references=kind == "room", two_level=kind == "instanced")


def _integrator(case):
    return api.IntegratorSettings(case["mode"], case["depth"], True, 3)


def _render(case, seed):
    return api.RenderSettings(case["width"], case["height"], case["spp"], 1 + seed)


def _rays(case, seed):
    """Unordered rays inside the unit room: uniform origins and directions."""
    rng = np.random.default_rng(seed)
    n = case["rays"]
    origins = rng.uniform((-0.45, 0.05, -0.45), (0.45, 0.95, 0.45), (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    far = rng.uniform(0.05, 1.5, n).astype(np.float32)
    keys = np.stack([np.full(n, 1 + seed), rng.integers(0, 1 << 20, n), np.arange(n)], 1)
    return origins, d.astype(np.float32), far, keys.astype(np.uint64)


def prepare(case, seed):
    call, kind = case["call"], case["scene"]
    state = {"case": case}
    if call == "batch":
        jobs = []
        for k in range(case["jobs"]):
            # Uneven like a queue: scene sizes over a factor of four, depths from 4 up.
            document = _document(kind, max(1000, case["triangles"] >> (k % 3)), 1000 * seed + k)
            integrator = api.IntegratorSettings(case["mode"], 4 + k % (case["depth"] - 3), True, 3)
            jobs.append(api.BatchJob(_build(kind, document), _render(case, seed + k), integrator))
        state["jobs"] = jobs
        return state
    document = _document(kind, case["triangles"], seed)
    if call == "build":
        state["snapshot"] = document.snapshot()
    else:
        state["scene"] = _build(kind, document)
    if call in ("nearest", "occluded", "paths"):
        state["rays"] = _rays(case, seed)
    if call == "paths" or call == "render":
        state["tracer"] = api.PathTracer(state["scene"], _integrator(case))
    if call == "session":
        state["session"] = api.RenderSession()
    if "width" in case:
        state["render"] = _render(case, seed)
    return state


# ---- the calls ----

def _with_counts(image, statistics):
    return {"image": image, "counts": {k: v for k, v in statistics.items()
                                       if not isinstance(v, dict) and "tests" not in k}}


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "render":
        return _with_counts(*state["tracer"].render(state["render"]))
    if call == "session":
        session = state["session"]
        session.start(state["scene"], state["render"], _integrator(case),
                      api.SessionSettings(batch_samples=4))
        session.wait()
        return _with_counts(session.result(), session.progress()["statistics"])
    if call == "batch":
        images, codes, _ = api.render_batch(state["jobs"])
        return {"images": images, "codes": codes}
    if call == "build":
        built = _build(case["scene"], state["snapshot"])
        out = _with_counts(*api.PathTracer(built, _integrator(case)).render(state["render"]))
        built.close()
        return out
    origins, directions, far, keys = state["rays"]
    if call == "nearest":
        hits, _ = state["scene"].intersect(origins, directions)
        return {name: hits[name] for name in hits.dtype.names}
    if call == "occluded":
        return state["scene"].occluded(origins, directions, 1e-5, far)[0]
    radiance, statistics = state["tracer"].trace(origins, directions, 1e-5, np.inf, keys)
    return _with_counts(radiance, statistics)


def work(case):
    """Geometry read and results written once; per ray one descent of a balanced tree (a box test
    of 24 flops per level, two triangle tests of 80), and two rays per vertex of a path that
    Russian roulette keeps to about four vertices."""
    triangles = case["triangles"]
    tests = 24 * math.log2(triangles) + 2 * 80
    scene_bytes = 36 * triangles
    if case["call"] in ("nearest", "occluded"):
        out = 40 if case["call"] == "nearest" else 1
        return {"bytes": case["rays"] * (32 + out) + scene_bytes, "flops": case["rays"] * tests}
    rays = 1 + 2 * min(case["depth"], 4)
    if case["call"] == "paths":
        return {"bytes": case["rays"] * (32 + 24 + 12) + scene_bytes,
                "flops": case["rays"] * rays * tests}
    jobs = case.get("jobs", 1)
    pixels = jobs * case["width"] * case["height"]
    return {"bytes": 12 * pixels + jobs * scene_bytes, "flops": pixels * case["spp"] * rays * tests}


# ---- the same in 64 bits ----
#
# Nearest hits by brute force, and the whole integrator for the Cornell box (diffuse walls, two
# area lights), on the same random streams. The other scenes' images have no value to be held to:
# their mirrors and glass turn the last bit of a direction into another path.

_EXACT_TESTS = 5e10  # ray-triangle pairs that take a few seconds


def exact(case, seed):
    if case["call"] == "nearest" and case["rays"] * case["triangles"] <= _EXACT_TESTS:
        return _exact_nearest(case, seed)
    samples = case.get("width", 1) * case.get("height", 1) * case.get("spp", 1)
    if (case["scene"] == "cornell" and case["mode"] == "mis" and samples <= 8_000_000
            and case["call"] in ("render", "session", "build", "paths")):
        return {"image": _exact_cornell(case, seed), "counts": None}
    return None


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _f64(a):
    return torch.as_tensor(np.asarray(a, np.float64), device=_device())


class _Triangles:
    """World-space triangles of a document in 64 bits: vertices, material and sidedness."""

    def __init__(self, document):
        vertices, material = [], []
        for o in document.objects:
            mesh = document.meshes[o.mesh]
            m = o.transform.matrix().astype(np.float64)
            p = mesh.positions.astype(np.float64)[mesh.corner_positions]
            vertices.append(p @ m[:3, :3] + m[3, :3])
            material.append(np.full(mesh.triangle_count, o.material))
        v = _f64(np.concatenate(vertices))
        self.material = torch.as_tensor(np.concatenate(material), device=_device())
        self.v0, self.e1, self.e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        self.cross = torch.cross(self.e1, self.e2, dim=1)
        double = torch.as_tensor([m.double_sided for m in document.materials], device=_device())
        self.one_sided = ~double[self.material]

    def nearest(self, o, d, lo, hi):
        """(distance, triangle, b1, b2) of the nearest hit per ray; infinite distance on a miss."""
        def dots(a, b):  # (rays, triangles) of ray-side and triangle-side vectors
            return a @ b.T

        det = -dots(d, self.cross)
        # With m = o x d: (o - v0) . (d x e) expands into products of ray and triangle vectors.
        m = torch.cross(o, d, dim=1)
        t = (dots(o, self.cross) - (self.v0 * self.cross).sum(1)) / det
        u = (dots(m, self.e2) + dots(d, torch.cross(self.v0, self.e2, dim=1))) / det
        v = (dots(m, self.e1) + dots(d, torch.cross(self.v0, self.e1, dim=1))) / -det
        ok = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= lo[:, None]) & (t <= hi[:, None])
        ok &= (det > 0) | ~self.one_sided
        t = torch.where(ok, t, torch.inf)
        best, index = t.min(1)
        return best, index, u.gather(1, index[:, None])[:, 0], v.gather(1, index[:, None])[:, 0]


def _exact_nearest(case, seed):
    triangles = _Triangles(_document(case["scene"], case["triangles"], seed))
    origins, directions, _, _ = _rays(case, seed)
    n = case["rays"]
    step = max(1, int(3e7) // triangles.v0.shape[0])
    distance, barycentric = np.zeros(n), np.zeros((n, 3))
    for k in range(0, n, step):
        o, d = _f64(origins[k:k + step]), _f64(directions[k:k + step])
        lo = torch.full_like(o[:, 0], float(np.float32(1e-5)))
        t, _, u, v = triangles.nearest(o, d, lo, torch.full_like(lo, torch.inf))
        hit = torch.isfinite(t)
        distance[k:k + step] = torch.where(hit, t, 0).cpu().numpy()
        b = torch.stack([1 - u - v, u, v], 1)
        barycentric[k:k + step] = torch.where(hit[:, None], b, 0).cpu().numpy()
    return {"distance": distance, "barycentric": barycentric, "front_face": None, "instance": None,
            "primitive": None, "triangle": None}


class _Streams:
    """The PCG32 streams of (seed, pixel, sample) keys in 64-bit integer tensors."""

    def __init__(self, seed, pixel, sample):
        def final(v):
            v = (v ^ self._shift(v, 30)) * self._signed(0xBF58476D1CE4E5B9)
            v = (v ^ self._shift(v, 27)) * self._signed(0x94D049BB133111EB)
            return v ^ self._shift(v, 31)

        start = final(seed ^ final(pixel + self._signed(0x9E3779B97F4A7C15)))
        sequence = final(sample + self._signed(0xD1B54A32D192ED03)) ^ final(pixel)
        self.increment = (sequence << 1) | 1
        self.state = torch.zeros_like(start)
        self._next()
        self.state = self.state + start
        self._next()

    @staticmethod
    def _signed(v):
        return v - (1 << 64) if v >= 1 << 63 else v

    @staticmethod
    def _shift(v, k):
        return (v >> k) & ((1 << (64 - k)) - 1)

    def _next(self):
        previous = self.state
        self.state = previous * 6364136223846793005 + self.increment
        shifted = self._shift(self._shift(previous, 18) ^ previous, 27) & 0xFFFFFFFF
        rotation = self._shift(previous, 59)
        return ((shifted >> rotation) | (shifted << ((32 - rotation) & 31))) & 0xFFFFFFFF

    def uniform(self):
        high, low = self._next() >> 5, self._next() >> 6
        return ((high << 26) | low).double() * 2.0 ** -53


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _dot(a, b):
    return (a * b).sum(-1)


def _heuristic(a, b):
    return torch.where(a + b > 0, a * a / (a * a + b * b).clamp_min(1e-300), 0.0)


def _disk(x, y):
    x, y = 2 * x - 1, 2 * y - 1
    wide = x.abs() > y.abs()
    radius = torch.where(wide, x, y)
    angle = torch.where(wide, math.pi / 4 * y / torch.where(wide, x, 1.0),
                        math.pi / 2 - math.pi / 4 * x / torch.where(wide | (y == 0), 1.0, y))
    return radius * angle.cos(), radius * angle.sin()


def _cornell_radiance(document, case, o, d, lo, hi, stream):
    """Radiance of a batch of paths through the diffuse, area-lit box (MIS, Russian roulette)."""
    tri = _Triangles(document)
    color = _f64([m.base_color for m in document.materials])
    emission = _f64([m.emission for m in document.materials])
    lights = (emission[tri.material].sum(1) > 0).nonzero()[:, 0]
    area = tri.cross.norm(dim=1) / 2
    normal = _unit(tri.cross)
    mass = area / area[lights].sum()  # one radiance, so power goes with the area
    cdf = torch.cumsum(mass[lights], 0)
    n = o.shape[0]
    radiance = torch.zeros_like(o)
    beta = torch.ones_like(o)
    alive = torch.ones(n, dtype=torch.bool, device=o.device)
    previous, pdf = o, torch.zeros_like(lo)

    def light_density(index, reference, point):
        to = point - reference
        cosine = _dot(normal[index], -_unit(to))
        return torch.where(cosine > 0, mass[index] * _dot(to, to) / (area[index] * cosine.abs()), 0.0)

    for depth in range(case["depth"] + 1):
        t, index, u, v = tri.nearest(o, d, lo, hi)
        alive = alive & torch.isfinite(t)
        t = torch.where(alive, t, 1.0)
        point = tri.v0[index] + u[:, None] * tri.e1[index] + v[:, None] * tri.e2[index]
        material = tri.material[index]
        weight = torch.ones_like(t) if depth == 0 else _heuristic(
            pdf, light_density(index, previous, point))
        radiance += torch.where(alive[:, None], beta * emission[material] * weight[:, None], 0.0)
        if depth == case["depth"]:
            break
        wo = -d
        nrm = normal[index]
        nrm = torch.where((_dot(nrm, wo) < 0)[:, None], -nrm, nrm)
        draws = [stream.uniform() for _ in range(6)]  # light, its point, component, direction
        # Next event: a point on one of the lights.
        pick = lights[torch.searchsorted(cdf, draws[0].contiguous(), right=True)
                      .clamp_max(len(lights) - 1)]
        root = draws[1].sqrt()
        target = (tri.v0[pick] + (root * (1 - draws[2]))[:, None] * tri.e1[pick]
                  + (root * draws[2])[:, None] * tri.e2[pick])
        density = light_density(pick, point, target)
        wi = _unit(target - point)
        cosine = _dot(wi, nrm)
        wanted = alive & (density > 0) & (cosine > 0)
        origin = point + 1e-9 * nrm
        length = (target - origin).norm(dim=1)
        blocked = torch.isfinite(tri.nearest(origin, _unit(target - origin), torch.zeros_like(length),
                                             length * (1 - 1e-6))[0])
        density = density.clamp_min(1e-300)
        gain = cosine / math.pi * _heuristic(density, cosine / math.pi) / density
        radiance += torch.where((wanted & ~blocked)[:, None],
                                beta * color[material] * emission[tri.material[pick]]
                                * gain[:, None], 0.0)
        # The next direction: cosine hemisphere about the normal.
        helper = torch.where((nrm[:, 2].abs() < 0.999)[:, None], _f64([0, 0, 1]), _f64([0, 1, 0]))
        tangent = _unit(torch.cross(helper, nrm, dim=1))
        bitangent = torch.cross(nrm, tangent, dim=1)
        x, y = _disk(draws[4], draws[5])
        z = (1 - x * x - y * y).clamp_min(0).sqrt()
        d = _unit(x[:, None] * tangent + y[:, None] * bitangent + z[:, None] * nrm)
        alive = alive & (z > 0)
        pdf = z / math.pi
        beta = beta * color[material]
        survival = stream.uniform()
        if depth + 1 >= 3:
            chance = beta.max(1).values.clamp(0.05, 0.95)
            alive = alive & (survival < chance)
            beta = beta / chance[:, None]
        previous, o = point, origin
        lo, hi = torch.zeros_like(lo), torch.full_like(hi, torch.inf)
    return radiance


def _exact_cornell(case, seed):
    document = _document("cornell", 36, seed)
    device = _device()
    chunk = 1 << 18

    def streams(key, pixel, sample):
        return _Streams(torch.full_like(pixel, key), pixel, sample)

    if case["call"] == "paths":
        origins, directions, _, keys = _rays(case, seed)
        k = torch.as_tensor(keys.astype(np.int64), device=device)
        lo = torch.full((len(origins),), float(np.float32(1e-5)), dtype=torch.float64, device=device)
        return _cornell_radiance(document, case, _f64(origins), _f64(directions), lo,
                                 torch.full_like(lo, torch.inf),
                                 streams(1 + seed, k[:, 1], k[:, 2])).cpu().numpy()
    width, height, spp = case["width"], case["height"], case["spp"]
    camera = document.camera
    position = _f64(camera.position)
    forward = _unit(_f64(camera.target) - position)
    right = _unit(torch.cross(forward, _f64(camera.up), dim=0))
    up = torch.cross(right, forward, dim=0)
    half = math.tan(math.radians(camera.vertical_fov_degrees) / 2)
    image = torch.zeros(height * width, 3, dtype=torch.float64, device=device)
    for sample in range(spp):
        for k in range(0, height * width, chunk):
            pixel = torch.arange(k, min(k + chunk, height * width), device=device)
            stream = streams(1 + seed, pixel, torch.full_like(pixel, sample))
            film = [stream.uniform() for _ in range(4)]  # pixel jitter, lens
            x = 2 * ((pixel % width) + film[0]) / width - 1
            y = 1 - 2 * ((pixel // width) + film[1]) / height
            d = _unit(forward + (x * width / height * half)[:, None] * right
                      + (y * half)[:, None] * up)
            cosine = _dot(d, forward)
            image[k:k + chunk] += _cornell_radiance(
                document, case, position.expand_as(d), d, camera.near_plane / cosine,
                camera.far_plane / cosine, stream)
    return (image / spp).reshape(height, width, 3).cpu().numpy()
