"""The work that a program built on this library has it do, as cases that can be timed: frames in the wavefront and the
plain form, single samples, rays, batched requests, an adaptive frame, the volume estimators and the adjoint, each
through the Python layer's public calls, from one small preview pass to the 12.3M-triangle frame.

A case is a dict of plain values; `prepare` makes what a program holds before the call (scenes loaded on the device,
pinned film arrays, ray and sample lists, parameters), `run` is one pass, `work` the bytes and operations a pass cannot
do without, `exact` a 64-bit answer where plain arithmetic gives one.
"""
import ctypes
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xpu2-foundation_b200"))
import x2  # noqa: E402
from x2 import diff  # noqa: E402

# Triangles of the generated scenes: the closed box (0), the fields of 12.3M (1), 1.16M (11), 771k (104) and 191k (108)
# triangles, the textured differentiable scene (4), and the medium in the box (33, with a grid of the case's own size).
TRIANGLES = {0: 34, 1: 12337152, 11: 1164288, 104: 771072, 108: 191488, 4: 247808, 33: 34}


def listed():
    return [
        # An interactive preview of a small scene: one sample a pixel, the film read back; launches and latency count.
        {"name": "box_preview", "entry": "wavefront", "scene": 0, "width": 256, "height": 256, "spp": 1},
        # The same scene's small frame in the drop-in lane's form, at a ragged size (partial tiles on two edges).
        {"name": "box_plain", "entry": "plain", "scene": 0, "width": 250, "height": 190, "spp": 16},
        # The headline frame: 12.3M triangles, 17 lights, 1920x1080, 64 samples a pixel.
        {"name": "field_frame", "entry": "wavefront", "scene": 1, "width": 1920, "height": 1080, "spp": 64},
        # A progressive viewer's pass over a field of 1.2M triangles: a few samples a pixel, an odd window size.
        {"name": "field_pass", "entry": "wavefront", "scene": 11, "width": 1283, "height": 719, "spp": 4},
        # A whole frame of a mid-sized field in the drop-in lane's form.
        {"name": "field_plain", "entry": "plain", "scene": 104, "width": 480, "height": 270, "spp": 64},
        # The per-sample entry: scattered (pixel, index) samples, as a caller of integrate() asks for them.
        {"name": "samples", "entry": "integrate", "scene": 108, "width": 240, "height": 135, "count": 60000},
        # The ray entry (closest hit and occlusion): a picking or visibility query of scattered rays.
        {"name": "rays", "entry": "rays", "scene": 108, "count": 262139},
        # Eight uneven requests (scene sizes, resolutions, samples and depths of their own) in one launch.
        {"name": "batch", "entry": "batch", "first": 0, "requests": 8, "spp_cap": 16},
        # An adaptive frame: passes with error estimates, region trees and masks between them.
        {"name": "adaptive", "entry": "adaptive", "scene": 0, "width": 250, "height": 190, "spp": 64, "target": 0.002},
        # A pass over the participating medium with the reference's march.
        {"name": "medium_march", "entry": "wavefront", "scene": 33, "width": 256, "height": 256, "spp": 4, "grid": 256, "estimator": 0},
        # The same medium by tracking.
        {"name": "medium_tracking", "entry": "wavefront", "scene": 33, "width": 512, "height": 512, "spp": 4, "grid": 256, "estimator": 1},
        # One optimisation step of the differentiable scene: the image, a loss, and its gradients.
        {"name": "adjoint", "entry": "adjoint", "scene": 4, "width": 512, "height": 512, "spp": 32, "adjoint_spp": 16},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    entry = rng.choice(["wavefront", "wavefront", "plain", "integrate", "rays", "batch", "adaptive", "march", "tracking", "adjoint"])
    if entry == "batch":
        return {"entry": "batch", "first": rng.randrange(40), "requests": rng.randint(1, 8), "spp_cap": _log(rng, 2, 16)}
    if entry == "rays":
        return {"entry": "rays", "scene": rng.choice([0, 11, 104, 108]), "count": _log(rng, 500, 1000000)}
    if entry == "integrate":
        return {"entry": "integrate", "scene": rng.choice([0, 104, 108]), "width": _log(rng, 64, 640), "height": _log(rng, 64, 480),
                "count": _log(rng, 500, 300000)}
    if entry in ("march", "tracking"):
        side = (40, 256) if entry == "march" else (64, 640)
        return {"entry": "wavefront", "scene": 33, "width": _log(rng, *side), "height": _log(rng, *side), "spp": _log(rng, 1, 6),
                "grid": rng.choice([32, 96, 128, 256]), "estimator": int(entry == "tracking")}
    if entry == "adaptive":
        return {"entry": "adaptive", "scene": rng.choice([0, 108]), "width": _log(rng, 64, 400), "height": _log(rng, 64, 300),
                "spp": _log(rng, 16, 128), "target": rng.choice([0.05, 0.01, 0.002])}
    if entry == "adjoint":
        return {"entry": "adjoint", "scene": 4, "width": _log(rng, 48, 640), "height": _log(rng, 48, 512), "spp": _log(rng, 2, 48),
                "adjoint_spp": _log(rng, 1, 24)}
    scene = rng.choice([0, 11, 104, 108])
    if entry == "plain":
        return {"entry": "plain", "scene": scene, "width": _log(rng, 32, 1280), "height": _log(rng, 32, 720), "spp": _log(rng, 1, 24)}
    return {"entry": "wavefront", "scene": scene, "width": _log(rng, 32, 1920), "height": _log(rng, 32, 1080), "spp": _log(rng, 1, 48)}


_CONTEXT = []


def _context():
    """The program's one device context."""
    if not _CONTEXT:
        _CONTEXT.append(x2.Context(0))
    return _CONTEXT[0]


def _resize(desc, cfg, width, height):
    """The config and the pinhole's raster at another image size (the vertical field of view stays)."""
    m = desc.camera.raster_to_camera
    s = m[0][0] * cfg.height / height
    m[0][0], m[1][1], m[3][0], m[3][1] = s, -s, -0.5 * width * s, 0.5 * height * s
    cfg.width, cfg.height = width, height


def _medium(desc, n, gen):
    """The medium's grids at n^3 voxels over its bounds: density in [0, 8] with its lowest 40 % empty, at half
    precision, from five octaves of noise, and emission on the hottest tenth. The arrays must outlive the scene's load."""
    def noise(octaves):
        v = torch.zeros((1, 1, n, n, n), device="cuda")
        for o in range(octaves):
            lattice = torch.rand((1, 1) + (min(n, 5 << o),) * 3, device="cuda", generator=gen) - 0.5
            v += 0.5 ** o * torch.nn.functional.interpolate(lattice, size=(n, n, n), mode="trilinear")
        return v.flatten()

    raw, heat = noise(5), noise(3)
    threshold, hot = (torch.kthvalue(raw, raw.numel() * 2 // 5).values, torch.kthvalue(heat, heat.numel() * 9 // 10).values)
    density = (8.0 * (raw - threshold).clamp(min=0) / (raw.max() - threshold)).half().float()
    power = torch.where((heat > hot) & (density > 0), 4.0 * (0.3 + 0.7 * (heat - hot) / (heat.max() - hot)) ** 4, torch.zeros_like(heat))
    emission = power[:, None] * torch.tensor([1.0, 0.55, 0.2], device="cuda")
    values = [density.cpu().numpy(), emission.contiguous().cpu().numpy()]
    volume = desc.volumes[0]
    lo, extent = volume.bound_lo[0], volume.bound_hi[0] - volume.bound_lo[0]
    volume.feature_size = extent / n
    for k, array in enumerate(values):
        g = desc.grids[k]
        for a in range(3):
            g.dims[a] = n
            g.world_to_index[a * 4 + a] = n / extent
            g.world_to_index[12 + a] = -lo * n / extent - 0.5
        g.values = array.ctypes.data_as(ctypes.POINTER(ctypes.c_float))
    return values


def _load(config_id, seed, width=None, height=None, generator_seed=None, grid=0, estimator=0, spp_cap=None):
    """A scene on the device: geometry and materials from the seed (generator_seed fixes them where they also set the
    work's size), the frame seed, and materials' and lights' colours moved a little by the seed."""
    source = x2.SyntheticScene(config_id, generator_seed if generator_seed is not None else seed + 1)
    desc, cfg = source.desc, source.config
    cfg.seed = seed & 0xffffffff
    if width:
        _resize(desc, cfg, width, height)
    if spp_cap:
        cfg.spp = min(cfg.spp, spp_cap)
    kept = None
    if grid:
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        kept = _medium(desc, grid, gen)
        cfg.max_depth = cfg.max_diffuse_depth = cfg.max_glossy_depth = cfg.max_mirror_depth = 64
        cfg.volume_estimator = estimator
    rng = np.random.default_rng(seed)
    for i in range(min(desc.material_count, 64)):
        m = desc.materials[i]
        for c in range(3):
            m.diffuse[c] *= float(rng.uniform(0.9, 1.0))
    for i in range(desc.light_count):
        scale = float(rng.uniform(0.9, 1.1))
        for c in range(3):
            desc.lights[i].radiance[c] *= scale
    scene = x2.Scene(_context(), desc, cfg)
    del kept
    return source, scene


def _film_arrays(cfg, odd=False):
    """Pinned film arrays that the program keeps across frames."""
    p = cfg.width * cfg.height
    sums = [torch.empty((p, 4), dtype=torch.float64, pin_memory=True).numpy() for _ in range(2 if odd else 1)]
    return (*sums, torch.empty(p, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32))


def _rays(n, seed):
    """Rays from inside and around the scene's bounds to points in them; half of them end at their target (visibility),
    half go on (picking)."""
    rng = np.random.default_rng(seed)
    rays = np.zeros((n, 8), np.float32)
    origin = rng.uniform(-1, 1, (n, 3))
    target = rng.uniform(-1, 1, (n, 3))
    return rays, origin, target, rng.random(n) < 0.5


def prepare(case, seed):
    entry = case["entry"]
    state = {"case": case}
    if entry == "batch":
        state["requests"] = []
        for k in range(case["requests"]):
            r = (case["first"] + k) % 48
            source, scene = _load(200 + r, seed + k, generator_seed=3, spp_cap=case["spp_cap"])
            state["requests"].append((scene, source.config.spp, _film_arrays(source.config)))
            source.free()
        return state
    source, scene = _load(case["scene"], seed, case.get("width"), case.get("height"), grid=case.get("grid", 0),
                          estimator=case.get("estimator", 0))
    cfg = source.config
    state["scene"] = scene
    if entry == "integrate":
        rng = np.random.default_rng(seed)
        state["pixels"] = rng.integers(0, cfg.width * cfg.height, case["count"], dtype=np.uint32)
        state["indices"] = rng.integers(0, 64, case["count"], dtype=np.uint32)
    elif entry == "rays":
        rays, origin, target, ends = _rays(case["count"], seed)
        half, centre = (np.array([0.95] * 3), np.zeros(3)) if case["scene"] == 0 else (np.array([11.0, 4.5, 11.0]), np.array([0.0, 4.0, 0.0]))
        direction = (target - origin) * half
        length = np.linalg.norm(direction, axis=1)
        rays[:, 0:3] = origin * half + centre
        rays[:, 3:6] = direction / length[:, None]
        rays[:, 6] = 0.0
        rays[:, 7] = np.where(ends, length * 0.999, 100.0)
        state["rays"] = rays
    elif entry == "adjoint":
        d = source.desc
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)

        def parameter(values, lo, hi):
            t = torch.tensor(np.array(values, np.float32), device="cuda")
            moved = t + 0.1 * (torch.rand(t.shape, device="cuda", generator=gen) - 0.5)
            return torch.where(t > 0, moved.clamp(lo, hi), t).requires_grad_(True)

        state["albedo"] = parameter([list(d.materials[m].diffuse) for m in range(d.material_count)], 0.02, 1.0)
        state["radiance"] = parameter([list(d.lights[i].radiance) for i in range(d.light_count)], 0.05, 30.0)
        state["roughness"] = parameter([d.materials[m].roughness for m in range(d.material_count)], 0.06, 0.9)
        state["texture"] = parameter(source.texture(0), 0.02, 0.95)
        state["target"] = torch.rand((cfg.height, cfg.width, 3), device="cuda", generator=gen)
    else:
        state["film"] = _film_arrays(cfg, odd=entry == "adaptive")
    source.free()
    return state


def run(state):
    case = state["case"]
    entry = case["entry"]
    if entry == "batch":
        _context().render_batch([(scene, 0, spp) for scene, spp, _ in state["requests"]])
        return [scene.film(out=film) for scene, _, film in state["requests"]]
    scene = state["scene"]
    if entry == "integrate":
        return scene.integrate(state["pixels"], state["indices"])
    if entry == "rays":
        return scene.trace_rays(state["rays"])
    if entry == "adaptive":
        result = scene.render_adaptive(4, case["spp"], case["target"])
        film = scene.film(odd=True, out=state["film"])
        return {"passes": result["passes"], "samples": result["samples"], "film": film}
    if entry == "adjoint":
        parameters = [state[k] for k in ("albedo", "radiance", "roughness", "texture")]
        image = diff.render(scene, parameters[0], parameters[1], 0, case["spp"], adjoint_first=case["spp"],
                            adjoint_count=case["adjoint_spp"], roughness=parameters[2], texture=parameters[3])
        loss = ((image - state["target"]) ** 2).sum()
        return [image.detach(), *torch.autograd.grad(loss, parameters)]
    scene.frame_begin(case["spp"])
    (scene.render_frame if entry == "plain" else scene.render_frame_wavefront)(0, case["spp"])
    scene.wait()
    return scene.film(out=state["film"])


# A path's rays and what each must do, for `work`: closest-hit and shadow rays a sample, as the scenes' light counts and
# depths make them, and the fewest 8-wide levels a ray descends (log8 of the triangles), each level eight boxes of
# twelve operations, then a triangle test. A medium's sample crosses its grid: about a lookup a voxel on the way.
_RAYS = {0: 7.0, 33: 12.0}


def _ray_flops(triangles):
    levels = max(1.0, float(np.log(triangles) / np.log(8.0)))
    return levels * 8 * 12 + 60


def work(case):
    entry = case["entry"]
    if entry == "batch":
        pixels, samples, triangles = 1e5 * case["requests"], 1e5 * case["requests"] * case["spp_cap"], 4e5 * case["requests"]
        return {"bytes": 48.0 * triangles + 36.0 * pixels, "flops": samples * 9.6 * _ray_flops(4e5)}
    triangles = TRIANGLES[case["scene"]]
    bytes_ = 48.0 * triangles
    per_sample = _RAYS.get(case["scene"], 9.6) * _ray_flops(triangles)
    if entry == "rays":
        # Scattered rays touch what they meet, not every triangle.
        return {"bytes": case["count"] * 44.0 + min(bytes_, 500.0 * case["count"]), "flops": case["count"] * 2 * _ray_flops(triangles)}
    if entry == "integrate":
        return {"bytes": case["count"] * 44.0 + min(bytes_, 2000.0 * case["count"]), "flops": case["count"] * per_sample}
    pixels = case["width"] * case["height"]
    if case.get("grid"):
        bytes_ += 16.0 * case["grid"] ** 3
        per_sample += 12.0 * case["grid"] * 20
    samples = pixels * (8 if entry == "adaptive" else case["spp"] + 1.5 * case.get("adjoint_spp", 0))
    film = (68.0 if entry == "adaptive" else 36.0) * pixels + (24.0 * 1024 * 1024 if entry == "adjoint" else 0.0)
    return {"bytes": bytes_ + film, "flops": samples * per_sample}


def exact(case, seed):
    """The rays' hit distances in 64 bits, every triangle against every ray (three Pluecker side products a pair). The
    other cases' outputs are sums over random walks whose every draw and decision is the library's own: plain arithmetic
    has no value for them."""
    if case["entry"] != "rays" or case["count"] * TRIANGLES[case["scene"]] > 6e10:
        return None
    source = x2.SyntheticScene(case["scene"], seed + 1)
    arrays = source.arrays()
    v = torch.tensor(arrays["vertices"].reshape(-1, 3), device="cuda").double()[torch.tensor(arrays["triangles"].reshape(-1, 3).astype(np.int64), device="cuda")]
    source.free()
    rays, origin, target, ends = _rays(case["count"], seed)
    half, centre = (np.array([0.95] * 3), np.zeros(3)) if case["scene"] == 0 else (np.array([11.0, 4.5, 11.0]), np.array([0.0, 4.0, 0.0]))
    direction = (target - origin) * half
    length = np.linalg.norm(direction, axis=1)
    o = torch.tensor((origin * half + centre).astype(np.float32), device="cuda").double()
    d = torch.tensor((direction / length[:, None]).astype(np.float32), device="cuda").double()
    far = torch.tensor(np.where(ends, length * 0.999, 100.0).astype(np.float32), device="cuda").double()
    t = torch.full_like(far, np.inf)
    ray = torch.cat([d, torch.linalg.cross(o, d)], 1)
    normal = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    # An edge's Pluecker coordinates, its moment first, so that a ray's side product is one dot product.
    edge = [torch.cat([torch.linalg.cross(v[:, k], v[:, (k + 1) % 3]), v[:, (k + 1) % 3] - v[:, k]], 1).T.contiguous() for k in range(3)]
    step = 1 << 14
    block = max(1, int(2e9 // (8 * step)))
    for a in range(0, len(v), step):
        for b in range(0, len(ray), block):
            r = ray[b:b + block]
            s = [r @ e[:, a:a + step] for e in edge]
            lo, hi = torch.minimum(torch.minimum(s[0], s[1]), s[2]), torch.maximum(torch.maximum(s[0], s[1]), s[2])
            i, j = torch.nonzero((lo >= 0) | (hi <= 0), as_tuple=True)
            i, j = i + b, j + a
            at = ((v[j, 0] - o[i]) * normal[j]).sum(1) / (d[i] * normal[j]).sum(1)
            ok = (at >= 0) & (at <= far[i])
            t.scatter_reduce_(0, i[ok], at[ok], "amin")
    t = torch.where(torch.isfinite(t), t, torch.zeros_like(t))  # a miss is given as 0
    return [None, t.cpu().numpy(), None]
