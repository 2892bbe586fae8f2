"""Performance cases of the renderer: the calls that programs make, from one ray pick to a 2.1 M triangle frame.

Every case is a plain dict; `kind` says which entry points a pass goes through:

  pick     DeviceRenderer.PickRay                                  (one ray, waits for the answer)
  frame    DeviceRenderer.RenderFrame                              (one accumulating frame, path tracing or another render mode)
  samples  DeviceRenderer.Reset + RenderSamples                    (an image of `spp` samples from scratch)
  train    DeviceRenderer.UpdateMaterials + RenderFrame + AdjointFrame   (one optimisation step's forward and backward)
  batch    BatchRenderer.Render + Image of every item              (many scenes as one wavefront)

Scenes are the package's seeded procedural ones; the seed changes geometry, materials, lights and random numbers.
"""
import math

import numpy as np
import torch

import trayracer_gb300 as tr

FLOAT = np.float64


def _case(name, kind, scene, width, height, **more):
    """All the fields that a case has, with what they are where a case does not say."""
    c = {"name": name, "kind": kind, "scene": scene, "width": width, "height": height,
         "size": 0,            # heightfield vertices a side, spheres of `spheres`, scenes of `batch`
         "ms": 1,              # samples a pixel of one wavefront frame
         "spp": 1,             # samples a pixel of a pass
         "depth": 16, "rr": 1 << 30,
         "graph": True,        # replayed as a CUDA graph
         "reference": False,   # the reference's own sampling
         "aovs": False,        # albedo and normal guides written too
         "mode": int(tr.RenderModes.PathTracing),
         "sky": False}
    c.update(more)
    return c


def listed():
    ao = int(tr.RenderModes.AmbientOcclusion)
    return [
        # a click in a viewport: what does this pixel show?
        _case("pick", "pick", "heightfield", 1280, 720, size=257),
        # a viewport that accumulates one sample a frame, with the renderer's default settings
        _case("preview_1spp", "frame", "cornell", 256, 256, ms=1, rr=1),
        # the small configuration, one eager frame: 256^2, 16 spp, 5 bounces, no Russian roulette
        _case("box_16spp", "frame", "cornell", 256, 256, ms=16, spp=16, depth=5, graph=False),
        # a comparison image in the reference's own sampling with denoiser guides, at an odd size
        _case("reference_aovs", "frame", "cornell_lambert", 317, 211, ms=2, spp=2, depth=16, rr=1, graph=False,
              reference=True, aovs=True),
        # a diagnostic image of terrain
        _case("ambient_occlusion", "frame", "heightfield", 1280, 720, size=385, depth=2, mode=ao),
        # an outdoor viewport under a sky
        _case("outdoor_sky", "frame", "outdoor", 960, 540, size=513, ms=4, spp=4, depth=8, rr=3, sky=True),
        # a textured room at an odd size, rendered to 16 samples
        _case("textured", "samples", "textured", 641, 479, ms=4, spp=16, depth=6, rr=3),
        # meshes placed by instances
        _case("instanced", "frame", "instanced", 1024, 768, ms=4, spp=4, depth=6, rr=3),
        # an optimisation step over 8 materials: 512^2, 32 spp, 6 bounces
        _case("train_box", "train", "cornell_disney", 512, 512, ms=32, spp=32, depth=6, rr=1 << 30),
        # an optimisation step over 800 materials and 4 M triangles, whose BVH outgrows the fp32 node layout
        _case("train_spheres", "train", "spheres", 1280, 720, size=800, ms=4, spp=4, depth=12, rr=3),
        # 16 scenes of uneven triangle count, resolution and sample count
        _case("batch_16", "batch", "batch", 0, 0, size=16, depth=6, rr=3),
        # the large configuration: a 2.1 M triangle heightfield, 1080p, 64 spp, 8 bounces
        _case("terrain_64spp", "samples", "heightfield", 1920, 1080, size=1024, ms=16, spp=64, depth=8, rr=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pick", "frame", "frame", "frame", "mode", "samples", "samples", "train", "batch"])
    width = _log(rng, 64, 1920)
    height = max(48, min(1080, int(width * rng.uniform(0.5, 1.0))))
    if rng.random() < 0.3:
        width, height = width // 8 * 8, height // 4 * 4
    n = _log(rng, 65, 900)
    if kind == "pick":
        return _unnamed("pick", rng.choice(["heightfield", "outdoor"]), width, height, size=n)
    if kind == "batch":
        return _unnamed("batch", "batch", 0, 0, size=rng.randint(3, 16), depth=rng.randint(3, 6), rr=rng.choice([3, 1 << 30]))
    if kind == "mode":
        return _unnamed("frame", rng.choice(["heightfield", "instanced", "cornell"]), width, height, size=n, depth=2,
                        mode=rng.choice([0, 1, 7, 8, 12]), graph=rng.random() < 0.5)
    scene = rng.choice({"frame": ["cornell", "cornell_lambert", "cornell_disney", "outdoor", "heightfield", "instanced", "textured"],
                        "samples": ["cornell", "cornell_disney", "outdoor", "heightfield", "instanced", "textured"],
                        "train": ["cornell", "cornell_disney", "cornell_disney", "heightfield", "spheres"]}[kind])
    ms = rng.choice([1, 2, 3, 4, 8, 16] if kind != "train" else [1, 4, 7, 16])
    if scene == "spheres":
        n = rng.randint(40, 500)
    while width * height * ms > 8_000_000:
        ms = max(1, ms // 2)
    frames = rng.choice([1, 2, 3, 4, 8]) if kind == "samples" else 1
    while frames > 1 and width * height * ms * frames > 24_000_000:
        frames -= 1
    spp = ms * frames
    reference = kind == "frame" and rng.random() < 0.25
    return _unnamed(kind, scene, width, height, size=n, ms=ms, spp=spp, depth=rng.randint(2, 12), rr=rng.choice([1, 3, 3, 1 << 30]),
                    graph=kind != "frame" or rng.random() < 0.6, reference=reference,
                    aovs=kind == "frame" and rng.random() < 0.3, sky=scene == "outdoor" and kind != "train" and rng.random() < 0.6)


def _unnamed(*args, **more):
    c = _case("", *args, **more)
    del c["name"]
    return c


def _scene(c, seed):
    w, h, s = c["width"], c["height"], c["scene"]
    if s == "cornell":
        return tr.cornell_box(seed=seed, width=w, height=h)
    if s == "cornell_lambert":
        return tr.cornell_box(seed=seed, width=w, height=h, wall_closure=tr.TR_CLOSURE_LAMBERT)
    if s == "cornell_disney":
        return tr.cornell_box(seed=seed, width=w, height=h, wall_closure=tr.TR_CLOSURE_DISNEY)
    if s == "textured":
        return tr.textured_cornell(seed=seed, width=w, height=h)
    if s == "instanced":
        return tr.instanced_cornell(seed=seed, width=w, height=h)
    if s == "heightfield":
        return tr.heightfield(n=c["size"], seed=seed, width=w, height=h)
    if s == "outdoor":  # terrain seen toward its horizon
        sc = tr.heightfield(n=c["size"], seed=seed, width=w, height=h)
        sc.camera.target = (0.0, 4.0, 0.0)
        return sc
    if s == "spheres":
        return tr.displaced_spheres(count=c["size"], n_emissive=max(1, c["size"] // 100), seed=seed, width=w, height=h,
                                    extent=40.0 * (c["size"] / 4096.0) ** (1.0 / 3.0))
    raise ValueError(s)


def _mix(count, seed):
    """The batching mix: triangle counts log-uniform in [1k, 500k], resolutions in 128^2 .. 1024^2, 4, 16 or 64 spp and
    1-16 lights, the same for every seed; the seed places the spheres and lights and draws the materials."""
    sizes = np.random.default_rng(11)
    return [tr.sphere_scene(seed * 1000 + k, int(round(1000 * 500.0 ** sizes.random())), res, res, spp, int(sizes.integers(1, 17)))
            for k, (res, spp) in enumerate(zip(sizes.choice([128, 256, 512, 1024], count).tolist(), sizes.choice([4, 16, 64], count).tolist()))]


class _DeviceArray:
    """A float4-per-pixel device buffer of the renderer, as torch takes it; the renderer lives as long as its views."""

    def __init__(self, owner, pointer, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (int(pointer), False), "version": 3}


def _view(renderer, name, shape):
    return torch.as_tensor(_DeviceArray(renderer, renderer.Buffers()[name], shape), device="cuda")


def _pixel(c, seed):
    r = np.random.default_rng([seed, 77])
    return int(r.integers(0, c["width"])), int(r.integers(c["height"] // 8, c["height"]))


def prepare(case, seed):
    c = dict(case)
    seed = int(seed) & 0x7FFFFFFF
    if c["kind"] == "batch":
        scenes = _mix(c["size"], seed % 1_000_003)
        b = tr.BatchRenderer(scenes)
        images = [torch.empty((s.height, s.width, 4), dtype=torch.float32, pin_memory=True).numpy() for s in scenes]
        ks = tr.KernelSettings(maxDepth=c["depth"], rrStart=c["rr"], seed=seed)
        return {"case": c, "batch": b, "settings": ks, "images": images}
    scene = _scene(c, seed)
    r = tr.DeviceRenderer(0)
    r.UpdateScene(scene)
    r.SetCamera(scene.camera)
    r.Resize((c["width"], c["height"]))
    if c["sky"]:
        rng = np.random.default_rng([seed, 5])
        r.SetSky(tr.SkySettings(sunDir=(float(rng.uniform(-0.5, 0.5)), 0.6, float(rng.uniform(0.2, 0.8))),
                                turbidity=float(rng.uniform(2.0, 6.0))))
    flags = (tr.TR_FLAG_REFERENCE_SAMPLING if c["reference"] else 0) | (tr.TR_FLAG_WRITE_AOVS if c["aovs"] else 0)
    ks = tr.KernelSettings(multiSample=c["ms"], maxDepth=c["depth"], seed=seed, rrStart=c["rr"], flags=flags, aoDist=1.5)
    r.SetSettings(ks)
    state = {"case": c, "renderer": r, "settings": ks, "mode": tr.RenderModes(c["mode"])}
    if c["kind"] == "pick":
        state["pixel"] = _pixel(c, seed)
        return state
    shape = (c["height"], c["width"], 4)
    for name in ("colors", "albedo", "normals") if c["aovs"] else ("colors",):
        state[name] = _view(r, name, shape)
    if c["kind"] == "train":
        state["materials"] = tr.perturbed_materials(scene.materials, seed=seed + 1, sigma=0.02)
        g = torch.Generator(device="cuda").manual_seed(seed)
        state["target"] = torch.rand(shape, generator=g, device="cuda") * 0.8
        state["grads"] = torch.zeros((scene.materials.shape[0], 9), device="cuda")
    return state


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "batch":
        b = state["batch"]
        b.Render(state["settings"])
        return [b.Image(i, out) for i, out in enumerate(state["images"])]
    r = state["renderer"]
    if kind == "pick":
        p = r.PickRay(state["pixel"])
        return {"origin": np.array(p.rayOrigin, np.float32), "direction": np.array(p.rayDir, np.float32),
                "distance": np.array([p.tmax], np.float32), "instance": int(p.instIx), "triangle": int(p.primIx)}
    if kind == "frame":
        r.RenderFrame(state["settings"], state["mode"], use_graph=c["graph"])
        return {k: state[k] for k in ("colors", "albedo", "normals") if k in state}
    if kind == "samples":
        r.Reset()
        r.RenderSamples(c["spp"])
        return {"colors": state["colors"]}
    # train: new parameters, the image, the gradient of 0.5 |image - target|^2
    r.UpdateMaterials(state["materials"])
    r.RenderFrame(state["settings"], use_graph=True)
    grads = state["grads"]
    grads.zero_()
    pixel_grad = state["colors"] - state["target"]
    r.AdjointFrame(pixel_grad.data_ptr(), 1.0 / c["ms"], grads.data_ptr())
    return {"colors": state["colors"], "grads": grads}


def _triangles(c):
    return {"heightfield": 2 * c["size"] ** 2, "outdoor": 2 * c["size"] ** 2, "spheres": 5000 * c["size"],
            "instanced": 400, "batch": 20_000}.get(c["scene"], 36)


def _image_work(c, samples, pixels, triangles):
    """Bytes: geometry (36 B of vertex positions and 16 B of indices and material a triangle) in, 16 B a pixel out
    (and the accumulator's 32 B). Operations: rays, each down a tree of 8 children a node (8 boxes of 24 operations a
    level) to two triangle tests of 45, and 400 operations to shade a hit."""
    levels = max(1.0, math.log(max(8, triangles), 8))
    ray = levels * 8 * 24 + 2 * 45
    closed = c["scene"].startswith(("cornell", "textured", "instanced"))
    if c["mode"] != int(tr.RenderModes.PathTracing):
        hits, rays = 1.0, min(2, c["depth"])
    else:  # closed rooms keep nearly every path; open scenes lose most after the first hit
        hits = min(c["depth"], 5.0 if closed and c["rr"] <= 3 else c["depth"] if closed else 1.3)
        rays = 2.0 * hits
    return {"bytes": triangles * 52.0 + pixels * 48.0, "flops": samples * (rays * ray + hits * 400.0)}


def work(case):
    c = case
    if c["kind"] == "pick":
        return {"bytes": 36.0 + 20 * 208.0, "flops": 20 * 8 * 24.0}
    if c["kind"] == "batch":
        pixels = c["size"] * 330_000.0  # the mean of 128^2 .. 1024^2
        return _image_work(c, pixels * 28.0, pixels, c["size"] * 80_000.0)
    pixels = c["width"] * c["height"]
    w = _image_work(c, pixels * float(c["spp"]), pixels, _triangles(c))
    if c["kind"] == "train":  # the replay traces the same rays again and evaluates two derivatives a vertex
        return {"bytes": 2 * w["bytes"] + pixels * 16.0, "flops": 3 * w["flops"]}
    return w


def exact(case, seed):
    """The picked ray and its distance in 64 bits: every triangle tested. Path-traced images have no such value here
    (their random decisions are made on rounded numbers)."""
    if case["kind"] != "pick":
        return None
    c = case
    seed = int(seed) & 0x7FFFFFFF
    scene = _scene(c, seed)
    x, y = _pixel(c, seed)
    cam = scene.camera

    def unit(v):
        return v / np.sqrt((v * v).sum())

    pos = np.asarray(cam.position, np.float32).astype(FLOAT)
    fwd = unit(np.asarray(cam.target, np.float32).astype(FLOAT) - pos)
    side = unit(np.cross(fwd, np.asarray(cam.up, FLOAT)))
    up = unit(np.cross(side, fwd))
    jitter, s = [], 0  # the linear congruential stream of state 0
    for _ in range(2):
        s = (1664525 * s + 1013904223) & 0xFFFFFFFF
        jitter.append((s & 0xFFFFFF) / float(1 << 24))
    t = math.tan(float(np.float32(cam.fov)) / 2)
    sx = (x + jitter[0]) / c["width"] * 2 - 1
    sy = ((c["height"] - y + jitter[1]) / c["height"] * 2 - 1) / (c["width"] / c["height"])
    d = unit(fwd + t * sx * side + t * sy * up)
    p = scene.positions.astype(FLOAT)
    i = scene.indices.astype(np.int64)
    v0 = p[i[:, 0]]
    e1, e2 = p[i[:, 1]] - v0, p[i[:, 2]] - v0
    q = np.cross(d, e2)
    det = (e1 * q).sum(1)
    ok = np.abs(det) > 0
    inv = 1.0 / np.where(ok, det, 1.0)
    tv = pos - v0
    u = (tv * q).sum(1) * inv
    r = np.cross(tv, e1)
    v = r @ d * inv
    dist = (e2 * r).sum(1) * inv
    ok &= (u >= 0) & (v >= 0) & (u + v <= 1) & (dist >= 1e-3)
    best = dist[ok].min() if ok.any() else None
    return {"origin": pos, "direction": d, "distance": None if best is None else np.array([best], FLOAT),
            "instance": None, "triangle": None}
