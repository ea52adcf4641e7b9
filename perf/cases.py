"""The work a user of this framework has it do, as cases that can be timed and compared.

Every case is one pass through the public entry points: renders (one frame at a time, as an editor's
view draws them, and many frames at once, as a still image is made), renders of translucent objects,
a batch of scenes in one pass, a differentiable render with its backward pass, and the per-query
entries (BSDF queries, multiscattering walks, ray queries).  Sizes come from the benchmark's
configurations and the tests' scenes; the seed moves the camera, the objects and the materials, never
a size, so every seed of a case costs the same.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from open_rendering_framework_b200 import _native as nat
from open_rendering_framework_b200 import diff
from open_rendering_framework_b200 import scene as sc
from open_rendering_framework_b200 import scenes

WALKS = tuple(sc.MSQ_OPS)
SCENES = ("single", "layered", "analytic", "sky")


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # an editor's thumbnail: the camera moves, one frame is drawn and read back for display
        {"name": "preview_96x64", "kind": "preview", "scene": "sky", "w": 96, "h": 64, "subdiv": 3, "depth": 6, "model": 0},
        # OptixScene::renderScene's loop at the window size of the single-scene configuration: one frame per call
        {"name": "frame_512x512", "kind": "render", "scene": "single", "w": 512, "h": 512, "frames": 1, "subdiv": 5, "depth": 8, "model": 0},
        # an odd-sized still of every layered material with the multiscattering model, a few frames
        {"name": "layered_301x203x6", "kind": "render", "scene": "layered", "w": 301, "h": 203, "frames": 6, "subdiv": 4, "depth": 8, "model": 2},
        # the single-scene configuration: 512 x 512, 64 samples per pixel, depth 8
        {"name": "still_512x512x64", "kind": "render", "scene": "single", "w": 512, "h": 512, "frames": 64, "subdiv": 6, "depth": 8, "model": 0},
        # one frame of a translucent object (directional dipole) at the reference's 500 probes per frame
        {"name": "skin_frame_203x151", "kind": "translucent", "w": 203, "h": 151, "frames": 1, "subdiv": 4, "probes": 500, "dipole": 1,
         "env": False, "depth": 6},
        # the subsurface configuration: standard dipole, 4,096 probes per frame, lit by an environment map
        {"name": "subsurface_512x512x4", "kind": "translucent", "w": 512, "h": 512, "frames": 4, "subdiv": 6, "probes": 4096, "dipole": 0,
         "env": True, "depth": 8},
        # the batched configuration, smaller: scenes of uneven size, resolution and material in one pass
        {"name": "batch_10_scenes", "kind": "batch", "scenes": 10, "w": 128, "frames": 4, "subdiv": 5},
        # the differentiable configuration: forward and backward of 256 x 256 at 16 samples per pixel
        {"name": "inverse_256x256x16", "kind": "inverse", "w": 256, "h": 256, "frames": 16, "subdiv": 5, "tex": 256, "probes": 500},
        # a tool's material preview: a few thousand BSDF queries
        {"name": "bsdf_4099", "kind": "bsdf", "n": 4099},
        # the BSDF-query configuration: 2^22 queries, half GGX and half Beckmann
        {"name": "bsdf_4M", "kind": "bsdf", "n": 1 << 22},
        # tabulating a rough dielectric with the multiscattering walk
        {"name": "walk_dielectric_500k", "kind": "walk", "op": "dielectric_sample", "dist": 1, "n": 500_009},
        # ray queries of a tool (picking, visibility): closest hit and any hit of incoherent rays
        {"name": "rays_1M", "kind": "rays", "n": 1_000_003, "subdiv": 5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("preview", "render", "render", "render", "translucent", "translucent", "batch", "inverse", "bsdf", "walk", "rays"))
    if kind == "preview":
        return {"kind": kind, "scene": rng.choice(SCENES), "w": _log(rng, 32, 320), "h": _log(rng, 32, 240), "subdiv": rng.randint(2, 5),
                "depth": rng.randint(4, 9), "model": rng.randint(0, 2)}
    if kind == "render":
        w, h = _log(rng, 64, 800), _log(rng, 48, 600)
        return {"kind": kind, "scene": rng.choice(SCENES), "w": w, "h": h, "frames": _log(rng, 1, max(1, min(64, (1 << 23) // (w * h)))),
                "subdiv": rng.randint(2, 6), "depth": rng.randint(4, 9), "model": rng.randint(0, 2)}
    if kind == "translucent":
        w, h = _log(rng, 48, 400), _log(rng, 48, 400)
        return {"kind": kind, "w": w, "h": h, "frames": rng.randint(1, 3), "subdiv": rng.randint(3, 5), "probes": _log(rng, 64, 2048),
                "dipole": rng.randint(0, 1), "env": rng.random() < 0.5, "depth": rng.randint(4, 8)}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 10), "w": _log(rng, 48, 128), "frames": rng.randint(1, 4), "subdiv": rng.randint(3, 5)}
    if kind == "inverse":
        return {"kind": kind, "w": _log(rng, 40, 256), "h": _log(rng, 40, 256), "frames": rng.randint(1, 12), "subdiv": rng.randint(3, 5),
                "tex": rng.choice((32, 64, 128, 256)), "probes": _log(rng, 100, 500)}
    if kind == "bsdf":
        return {"kind": kind, "n": _log(rng, 1000, 1 << 22)}
    if kind == "walk":
        return {"kind": kind, "op": rng.choice(WALKS), "dist": rng.randint(0, 1), "n": _log(rng, 1000, 500_000)}
    return {"kind": kind, "n": _log(rng, 1000, 1_000_000), "subdiv": rng.randint(3, 6)}


# ---------------------------------------------------------------- scenes
@functools.lru_cache(maxsize=None)
def _sphere(subdiv):
    return scenes.icosphere(subdiv)


@functools.lru_cache(maxsize=None)
def _sky(w, h):
    return scenes.sky_envmap(w, h, sun_peak=5.0e4 if w >= 1024 else 2.0e3, sun_sigma_deg=1.0 if w >= 1024 else 6.0)


def _env(rng, w, h):
    return sc.EnvMapBackground(np.ascontiguousarray(_sky(w, h) * np.float32(rng.uniform(0.7, 1.3))))


def _ball(subdiv, radius, center, material, rng, amplitude=0.0):
    """A sphere of 20 * 4^subdiv triangles, smoothly bumped by the seed when amplitude > 0."""
    p, vi, n, _ = _sphere(subdiv)
    p = p.astype(np.float64)
    if amplitude:
        k, ph = rng.uniform(2.0, 5.0, (3, 3)), rng.uniform(0.0, 2.0 * np.pi, 3)
        p = p * (1.0 + amplitude * np.sin(p @ k + ph).mean(axis=1, keepdims=True))
    return sc.Mesh((p * radius + np.asarray(center)).astype(np.float32), vi, material, n, vi)


def _grid(n, rng, material):
    t = np.linspace(-0.6, 0.6, n + 1)
    X, Z = np.meshgrid(t, t, indexing="ij")
    a, b = rng.uniform(4.0, 9.0, 2)
    Y = -0.35 + 0.08 * np.sin(a * X) * np.cos(b * Z)
    N = np.stack([-0.08 * a * np.cos(a * X) * np.cos(b * Z), np.ones_like(X), 0.08 * b * np.sin(a * X) * np.sin(b * Z)], -1)
    N /= np.linalg.norm(N, axis=-1, keepdims=True)
    i = np.arange((n + 1) ** 2).reshape(n + 1, n + 1)
    q = [i[:-1, :-1].ravel(), i[1:, :-1].ravel(), i[1:, 1:].ravel(), i[:-1, 1:].ravel()]
    tri = np.concatenate([np.stack([q[0], q[2], q[1]], 1), np.stack([q[0], q[3], q[2]], 1)]).astype(np.int32)
    return sc.Mesh(np.stack([X, Y, Z], -1).reshape(-1, 3), tri, material, N.reshape(-1, 3), tri)


def _room(rng, albedo=0.7):
    p, i = scenes.box()
    c = np.clip(albedo + rng.uniform(-0.1, 0.1, 3), 0.05, 0.95)
    return sc.Mesh(p, i, sc.DiffuseMaterial(tuple(c)))


def _quad(rng, size=0.25):
    p, i = scenes.quad_light((rng.uniform(-0.2, 0.2), 0.99, rng.uniform(-0.2, 0.2)), size)
    return sc.TriangleAreaLight(p, i, tuple(rng.uniform(12.0, 18.0, 3)))


def _near(rng, x, y, z):
    return tuple(np.array([x, y, z]) + rng.uniform(-0.03, 0.03, 3))


def _indoor_camera(rng, c):
    return sc.PinholeCamera(eye=_near(rng, 0.0, 0.0, 0.9), lookat=_near(rng, 0.0, -0.1, -1.0), up=(0.0, 1.0, 0.0), vfov=60.0, width=c["w"], height=c["h"])


def _conductor(rng, model, dist=sc.GGX_DISTRIBUTION):
    a = float(rng.uniform(0.15, 0.3))
    return sc.MetallicMaterial(ior=((0.2, 3.9), (0.55, 3.15), (0.9, 2.4)), roughness=(a, a), microfacet_model=model, normal_distribution=dist)


def _dielectric(rng, model):
    return sc.RoughTransparentMaterial(ior=float(rng.uniform(1.4, 1.6)), roughness=float(rng.uniform(0.08, 0.15)), microfacet_model=model,
                                       normal_distribution=sc.BECKMANN_DISTRIBUTION)


def _scene(c, rng):
    """The scene of a "preview" or "render" case."""
    s, sub, model = c["scene"], c["subdiv"], c["model"]
    integrator = sc.PathTracer(max_depth=c["depth"], scene_epsilon=1e-4, rr_start_depth=3)
    if s == "sky":  # an open scene: floor, conductor and dielectric under the sky, which is also the light
        floor = sc.Mesh(np.array([(-3, -1, -3), (3, -1, -3), (3, -1, 3), (-3, -1, 3)], np.float32), np.array([(0, 2, 1), (0, 3, 2)], np.int32),
                        sc.DiffuseMaterial(tuple(rng.uniform(0.4, 0.7, 3))))
        meshes = [floor, _ball(sub, 0.5, _near(rng, -0.6, -0.5, 0.0), _conductor(rng, model), rng),
                  _ball(max(1, sub - 1), 0.5, _near(rng, 0.6, -0.5, 0.2), _dielectric(rng, model), rng)]
        camera = sc.PinholeCamera(eye=_near(rng, 0.0, 0.3, 2.2), lookat=(0.0, -0.3, 0.0), up=(0.0, 1.0, 0.0), vfov=45.0, width=c["w"], height=c["h"])
        return sc.SceneData(integrator, camera, _env(rng, 256, 128), meshes, [sc.EnvMapLight()])
    camera, background = _indoor_camera(rng, c), sc.ConstantBackground((0.0, 0.0, 0.0))
    if s == "single":
        meshes = [_room(rng), _ball(sub, 0.3, _near(rng, -0.45, -0.65, -0.3), _conductor(rng, model), rng),
                  _ball(max(1, sub - 1), 0.3, _near(rng, 0.45, -0.65, 0.1), _dielectric(rng, model), rng)]
        return sc.SceneData(integrator, camera, background, meshes, [_quad(rng)])
    if s == "layered":
        a = float(rng.uniform(0.2, 0.4))
        rough = sc.RoughDiffuseMaterial(color=tuple(rng.uniform(0.2, 0.8, 3)), ior=1.4, roughness=(a, a), microfacet_model=model,
                                        normal_distribution=sc.BECKMANN_DISTRIBUTION)
        meshes = [_room(rng), _ball(sub, 0.28, _near(rng, -0.48, -0.45, -0.45), sc.LambertianInterfaceMaterial(tuple(rng.uniform(0.2, 0.8, 3)), 1.5), rng),
                  _ball(sub, 0.28, _near(rng, 0.08, -0.45, -0.6), rough, rng),
                  _ball(sub, 0.25, _near(rng, 0.45, -0.4, -0.2), sc.TransparentMaterial(ior=1.5, glass_absorption=(0.5, 0.2, 0.1)), rng)]
        return sc.SceneData(integrator, camera, background, meshes, [_quad(rng)])
    meshes = [_room(rng), _ball(sub, 0.28, _near(rng, -0.4, -0.6, -0.4), _conductor(rng, model), rng),
              _ball(sub, 0.25, _near(rng, 0.4, -0.65, -0.1), sc.LambertianInterfaceMaterial((0.3, 0.5, 0.7), 1.5), rng)]
    lights = [sc.DiskAreaLight(position=_near(rng, 0.0, 0.9, 0.0), radiance=(8.0, 8.0, 7.0), radius=0.2, theta=180.0, phi=0.0),
              sc.SphericalLight(position=_near(rng, 0.3, 0.3, -0.4), radiance=(20.0, 18.0, 15.0), radius=0.08)]
    return sc.SceneData(integrator, camera, background, meshes, lights)


def _translucent(c, rng):
    s, a = rng.uniform(0.5, 3.0, 3), rng.uniform(0.001, 0.05, 3)
    integrator = sc.PathTracer(max_depth=c["depth"], scene_epsilon=1e-4)
    if c["env"]:
        mat = sc.TranslucentMaterial(scattering=tuple(s), absorption=tuple(a), ior=1.3, scale=100.0, dipole_model=c["dipole"])
        camera = sc.PinholeCamera(eye=_near(rng, 0.0, 0.35, 2.0), lookat=(0.0, 0.0, 0.0), up=(0.0, 1.0, 0.0), vfov=36.0, width=c["w"], height=c["h"])
        return sc.SceneData(integrator, camera, _env(rng, 2048, 1024), [_ball(c["subdiv"], 0.5, (0.0, 0.0, 0.0), mat, rng, 0.04)], [sc.EnvMapLight()],
                            probe_samples=c["probes"])
    mat = sc.TranslucentMaterial(scattering=tuple(s), absorption=tuple(4.0 * a), ior=1.3, scale=10.0, dipole_model=c["dipole"])
    meshes = [_room(rng), _ball(c["subdiv"], 0.35, _near(rng, -0.2, -0.55, -0.2), mat, rng, 0.04)]
    return sc.SceneData(integrator, _indoor_camera(rng, c), sc.ConstantBackground((0.0, 0.0, 0.0)), meshes, [_quad(rng, 0.5)], probe_samples=c["probes"])


def _batch_item(c, k, rng):
    """Scene k of a batch and its frames: material, mesh, resolution and frames follow k, as unevenly as the
    batched configuration draws them."""
    res, frames = c["w"] * (1, 2, 1, 4)[k % 4], c["frames"] * (1, 2, 4, 1, 3)[k % 5]
    kind = scenes.BATCH_MATERIALS[k % 5]
    if kind == "diffuse":
        mat = sc.DiffuseMaterial(tuple(rng.uniform(0.3, 0.9, 3)))
    elif kind == "ggx":
        mat = _conductor(rng, sc.VISIBLE_NORMALS_MODEL)
    elif kind == "beckmann":
        mat = _conductor(rng, sc.WALTER_MODEL, sc.BECKMANN_DISTRIBUTION)
    elif kind == "rough_dielectric":
        mat = _dielectric(rng, sc.WALTER_MODEL)
    else:
        mat = sc.TranslucentMaterial(scattering=tuple(rng.uniform(0.5, 3.0, 3)), absorption=tuple(rng.uniform(0.001, 0.05, 3)), ior=1.3, scale=100.0)
    sub = max(2, c["subdiv"] - k % 3)
    mesh = _grid(3 * 2 ** sub, rng, mat) if k % 2 else _ball(sub, 0.4, (0.0, 0.0, 0.0), mat, rng, 0.04)
    floor = sc.Mesh(np.array([(-4, -0.45, -4), (4, -0.45, -4), (4, -0.45, 4), (-4, -0.45, 4)], np.float32), np.array([(0, 2, 1), (0, 3, 2)], np.int32),
                    sc.DiffuseMaterial((0.5, 0.5, 0.5)))
    az = rng.uniform(0.0, 2.0 * np.pi)
    camera = sc.PinholeCamera(eye=(2.0 * np.sin(az), 0.8, 2.0 * np.cos(az)), lookat=(0.0, -0.1, 0.0), up=(0.0, 1.0, 0.0), vfov=40.0, width=res, height=res)
    data = sc.SceneData(sc.PathTracer(max_depth=8, scene_epsilon=1e-4, rr_start_depth=3), camera, _env(rng, 128, 64), [mesh, floor], [sc.EnvMapLight()],
                        probe_samples=500)
    return data, frames


def _inverse(c, rng):
    diffuse, t = sc.DiffuseMaterial((0.7, 0.7, 0.7)), c["tex"]
    diffuse.setTexture(np.full((t, t, 3), 0.5, np.float32), (0.0, 0.0, 0.0))
    center = (-0.45, -0.65, -0.3)
    metal = _conductor(rng, sc.WALTER_MODEL)
    metal.setTexture(np.full((t, t), 0.5, np.float32), center)
    skin = sc.TranslucentMaterial(scattering=(0.5,) * 3, absorption=(0.5,) * 3, ior=1.3, scale=10.0)
    p, i = scenes.box()
    meshes = [sc.Mesh(p, i, diffuse), _ball(c["subdiv"], 0.3, center, metal, rng), _ball(c["subdiv"], 0.3, _near(rng, 0.45, -0.65, 0.1), skin, rng)]
    data = sc.SceneData(sc.PathTracer(max_depth=6, scene_epsilon=1e-4, rr_start_depth=3), _indoor_camera(rng, c), sc.ConstantBackground((0.0, 0.0, 0.0)),
                        meshes, [_quad(rng)], probe_samples=c["probes"])
    return data, (diffuse, metal, skin)


# ---------------------------------------------------------------- inputs
def _image(c):
    return torch.empty((c["h"], c["w"], 4), dtype=torch.float32, device="cuda")


def _directions(n, g, lo=-1.0):
    """Unit vectors with z uniform in [lo, 1], three rows of n."""
    z = lo + (1.0 - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    p = 2.0 * math.pi * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    r = torch.sqrt(1.0 - z * z)
    return torch.stack([r * torch.cos(p), r * torch.sin(p), z]).float().contiguous()


def _ray_scene(case, seed):
    c = dict(case, scene="single", w=64, h=64, depth=8, model=0)
    return _scene(c, np.random.default_rng(seed))


def _rays(case, seed):
    """Rays from points inside the room in every direction (origin and tmin, direction and tmax)."""
    g = torch.Generator("cuda").manual_seed(seed)
    n = case["n"]
    o = torch.empty((n, 4), device="cuda")
    o[:, :3] = 1.8 * torch.rand((n, 3), generator=g, device="cuda") - 0.9
    o[:, 3] = 1e-4
    d = torch.full((n, 4), 1e27, device="cuda")
    d[:, :3] = _directions(n, g).T
    any_d = d.clone()
    any_d[:, 3] = 0.05 + 1.5 * torch.rand(n, generator=g, device="cuda")  # visibility over a distance
    return o, d, any_d


def _bsdf_inputs(case, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    wo = _directions(case["n"], g, lo=0.01)
    alpha = 0.05 + 0.95 * torch.rand(case["n"], generator=g, device="cuda")
    return wo, alpha, 1000 * (seed % 1000)  # the batch's first global index: the draws are seeded by it


def prepare(case, seed):
    c, rng, kind = case, np.random.default_rng(seed), case["kind"]
    if kind in ("preview", "render", "translucent"):
        data = _translucent(c, rng) if kind == "translucent" else _scene(c, rng)
        return {"case": c, "R": sc.Renderer(data), "out": None if kind == "preview" else _image(c)}
    if kind == "batch":
        items = [_batch_item(c, k, rng) for k in range(c["scenes"])]
        rs = [sc.Renderer(d) for d, _ in items]
        return {"case": c, "rs": rs, "B": sc.Batch(rs, [f for _, f in items]),
                "out": [torch.empty((d.camera.height, d.camera.width, 4), device="cuda") for d, _ in items]}
    if kind == "inverse":
        data, mats = _inverse(c, rng)
        g, t = torch.Generator("cuda").manual_seed(seed), c["tex"]
        p = [torch.rand(s, generator=g, device="cuda") * 0.8 + 0.1 for s in ((t, t, 3), (t, t), (6,))]
        target = torch.rand((c["h"], c["w"], 3), generator=g, device="cuda")
        return {"case": c, "S": diff.DiffScene(data, *mats), "params": [x.requires_grad_() for x in p], "target": target}
    n = case["n"]
    if kind == "bsdf":
        wo, alpha, first = _bsdf_inputs(case, seed)
        return {"case": c, "wo": wo, "alpha": alpha, "first": first, "wi": torch.empty_like(wo), "f": torch.empty_like(alpha),
                "pdf": torch.empty_like(alpha), "F": torch.empty_like(alpha)}
    if kind == "walk":
        g = torch.Generator("cuda").manual_seed(seed)
        both = case["op"] == "dielectric_eval"
        wi, wo = _directions(n, g, lo=0.02), _directions(n, g, lo=-0.98 if both else 0.02)
        m = sc.MicrofacetBatch(op=sc.MSQ_OPS[case["op"]], normal_distribution=case["dist"], normal=(0.0, 0.0, 1.0), eta=1.0 / 1.5,
                               ior=(0.2, 3.9, 0.55, 3.15, 0.9, 2.4), rho=(0.8, 0.6, 0.4))
        seeds = torch.randint(0, 2 ** 31 - 1, (n,), generator=g, device="cuda", dtype=torch.int32)
        return {"case": c, "m": m, "wi": wi, "wo": wo, "alpha": 0.05 + 0.95 * torch.rand(n, generator=g, device="cuda"), "seed0": seeds,
                "seed": seeds.clone(), "order": torch.zeros_like(seeds), "out": torch.empty_like(wi), "weight": torch.empty_like(wi)}
    o, d, any_d = _rays(case, seed)
    return {"case": c, "R": sc.Renderer(_ray_scene(case, seed)), "o": o, "d": d, "any_d": any_d, "prim": torch.empty(n, dtype=torch.int32, device="cuda"),
            "t": torch.empty(n, device="cuda"), "bary": torch.empty((n, 2), device="cuda"), "hit": torch.empty(n, dtype=torch.int32, device="cuda")}


# ---------------------------------------------------------------- one pass
def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "preview":
        R = state["R"]
        R.apply_camera()
        R.renderScene()
        return R.readback()
    if kind in ("render", "translucent"):
        R = state["R"]
        R.frame = 0
        R.render(c["frames"])
        nat.call("pt_readback_device", R.ctx, state["out"].data_ptr())
        return state["out"]
    if kind == "batch":
        for R in state["rs"]:
            R.apply_camera()  # the images start over
        state["B"].render()
        for R, out in zip(state["rs"], state["out"]):
            nat.call("pt_readback_device", R.ctx, out.data_ptr())
        return state["out"]
    if kind == "inverse":
        image = diff.render(state["S"], c["frames"], *state["params"])
        loss = ((image - state["target"]) ** 2).sum()
        grads = torch.autograd.grad(loss, state["params"])
        return {"image": image.detach(), "albedo": grads[0], "roughness": grads[1], "sigma": grads[2]}
    if kind == "bsdf":
        s, n = state, c["n"]
        nat.call("pt_bsdf_queries", s["wo"].data_ptr(), s["alpha"].data_ptr(), n, s["first"], s["first"] + n // 2, 1.0 / 1.5, s["wi"].data_ptr(),
                 s["f"].data_ptr(), s["pdf"].data_ptr(), s["F"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"wi": s["wi"], "f": s["f"], "pdf": s["pdf"], "F": s["F"]}
    if kind == "walk":
        s = state
        s["seed"].copy_(s["seed0"])
        s["order"].zero_()
        nat.call("pt_microfacet_queries", ctypes.byref(s["m"]), s["wi"].data_ptr(), s["wo"].data_ptr(), s["alpha"].data_ptr(), s["seed"].data_ptr(),
                 s["order"].data_ptr(), c["n"], s["out"].data_ptr(), s["weight"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"out": s["out"], "weight": s["weight"], "seed": s["seed"], "order": s["order"]}
    s = state
    nat.call("pt_trace_closest", s["R"].ctx, s["o"].data_ptr(), s["d"].data_ptr(), c["n"], s["prim"].data_ptr(), s["t"].data_ptr(), s["bary"].data_ptr())
    nat.call("pt_trace_any", s["R"].ctx, s["o"].data_ptr(), s["any_d"].data_ptr(), c["n"], s["hit"].data_ptr())
    return {"prim": s["prim"], "t": s["t"], "bary": s["bary"], "hit": s["hit"]}


# ---------------------------------------------------------------- what a pass cannot do without
# Operations of one step of a path (a closest-hit ray, the shading of its hit with about seven 16-round
# draws, and a shadow ray: about 3,000 integer and floating operations), of one (hit, probe) pair of a
# dipole gather (one MD5 draw, a distance, an exponential), and of one query.
_STEP, _PAIR, _BSDF, _WALK, _RAY = 3000.0, 230.0, 1500.0, 4000.0, 1000.0


def _triangles(c):
    return 20 * 4 ** c.get("subdiv", 0)


def work(case):
    c, kind = case, case["kind"]
    if kind in ("preview", "render"):
        paths = c["w"] * c["h"] * c.get("frames", 1)
        return {"bytes": 16.0 * c["w"] * c["h"] + 100.0 * _triangles(c), "flops": paths * _STEP * (2.5 if c["scene"] == "sky" else 0.7 * c["depth"])}
    if kind == "translucent":
        paths, probes = c["w"] * c["h"] * c["frames"], c["probes"] * c["frames"]
        env = 16.0 * 2048 * 1024 if c["env"] else 0.0
        entries = 0.45 if c["env"] else 0.12  # gathers per path; three quarters of the probes are lit
        return {"bytes": 16.0 * c["w"] * c["h"] + 100.0 * _triangles(c) + env,
                "flops": (paths + probes) * _STEP * 2.5 + paths * entries * 0.75 * c["probes"] * _PAIR}
    if kind == "batch":
        items = [((1, 2, 1, 4)[k % 4] * c["w"], c["frames"] * (1, 2, 4, 1, 3)[k % 5]) for k in range(c["scenes"])]
        return {"bytes": sum(16.0 * r * r for r, _ in items) + 100.0 * _triangles(c) * c["scenes"], "flops": sum(r * r * f for r, f in items) * _STEP * 2.2}
    if kind == "inverse":
        paths = c["w"] * c["h"] * c["frames"]
        return {"bytes": 28.0 * c["w"] * c["h"] + 32.0 * c["tex"] ** 2 + 200.0 * _triangles(c),
                "flops": 2.0 * paths * (_STEP * 4.7 + 0.137 * 0.6 * c["probes"] * _PAIR)}
    n = c["n"]
    if kind == "bsdf":
        return {"bytes": 40.0 * n, "flops": _BSDF * n}
    if kind == "walk":
        return {"bytes": 60.0 * n, "flops": _WALK * n}
    return {"bytes": 80.0 * n + 100.0 * _triangles(c), "flops": 2.0 * _RAY * n}


# ---------------------------------------------------------------- the results in 64 bits
def _tea(v0, v1):
    """tea<16> on int64 tensors holding 32-bit words."""
    M, s = 0xFFFFFFFF, 0
    for _ in range(16):
        s = (s + 0x9E3779B9) & M
        v0 = (v0 + ((((v1 << 4) + 0xA341316C) & M) ^ ((v1 + s) & M) ^ (((v1 >> 5) + 0xC8013EA4) & M))) & M
        v1 = (v1 + ((((v0 << 4) + 0xAD90777D) & M) ^ ((v0 + s) & M) ^ (((v0 >> 5) + 0x7E95761E) & M))) & M
    return v0


def _draw(s):
    s = _tea(s, torch.full_like(s, 100))
    return s, ((s & 0x7FFFFFFF).float() / 2147483648.0).double()


def _beckmann_slopes(th, z1, z2):
    si, co = torch.sin(th), torch.cos(th)
    a = co / si
    c = 1.0 / (0.5 * (torch.erf(a) + 1.0) * co + 0.5 / math.sqrt(math.pi) * si * torch.exp(-a * a))
    lo = torch.full_like(th, -0.9999)
    hi = torch.maximum(lo, torch.erf(a))
    cur = 0.5 * (lo + hi)
    live = torch.ones_like(th, dtype=torch.bool)
    for _ in range(256):
        live = live & (hi - lo > 1e-5)
        if not bool(live.any()):
            break
        cur = torch.where(live & ~((cur >= lo) & (cur <= hi)), 0.5 * (lo + hi), cur)
        s = torch.erfinv(cur)
        cdf = torch.where(s >= a, torch.ones_like(s), c * (0.5 / math.sqrt(math.pi) * si * torch.exp(-s * s) + co * (0.5 + 0.5 * torch.erf(s))))
        d = cdf - z1
        live = live & ~(d.abs() < 1e-5)
        stop = torch.where(d > 0, hi == cur, lo == cur)
        live = live & ~stop
        hi = torch.where(live & (d > 0), cur, hi)
        lo = torch.where(live & ~(d > 0), cur, lo)
        cur = torch.where(live, cur - d / (0.5 * c * co - 0.5 * c * si * s), cur)
    return torch.erfinv(torch.minimum(hi, torch.maximum(lo, cur))), torch.erfinv(2.0 * z2 - 1.0)


def _ggx_slopes(th, z1, z2):
    si, co = torch.sin(th), torch.cos(th).clamp_min(1e-7)
    t = si / co
    A = 2.0 * z1 / co * 0.5 * (co + 1.0) - 1.0
    m = 1.0 / (A * A - 1.0)
    D = torch.sqrt((t * t * m * m - (A * A - t * t) * m).clamp_min(0.0))
    s1, s2 = t * m - D, t * m + D
    x = torch.where((A < 0) | (s2 > 1.0 / t), s1, s2)
    S = torch.where(z2 > 0.5, 1.0, -1.0)
    z = 2.0 * (z2 - 0.5).abs()
    q = (z * (z * (z * 0.27385 - 0.73369) + 0.46341)) / (z * (z * (z * 0.093073 + 0.309420) - 1.0) + 0.597999)
    return x, S * q * torch.sqrt(1.0 + x * x)


def _bsdf_exact(case, seed):
    wo, alpha, first = _bsdf_inputs(case, seed)
    n, a, w = case["n"], alpha.double(), wo.double()
    k = torch.arange(n, device="cuda", dtype=torch.int64)
    ggx = k < n // 2
    s = _tea((first + k) & 0xFFFFFFFF, torch.zeros_like(k))
    s, u1 = _draw(s)
    s, u2 = _draw(s)
    unit = lambda v: v / v.norm(dim=0)  # noqa: E731
    loc = unit(torch.stack([-w[0], -w[1], w[2]]))
    v = unit(torch.stack([a * loc[0], a * loc[1], loc[2]]))
    th, ph = torch.acos(v[2].clamp(-1.0, 1.0)), torch.atan2(v[1], v[0])
    gx, gy = _ggx_slopes(th, u1, u2)
    bx, by = _beckmann_slopes(th, u1, u2)
    x, y = torch.where(ggx, gx, bx), torch.where(ggx, gy, by)
    sx, sy = a * (torch.cos(ph) * x - torch.sin(ph) * y), a * (torch.sin(ph) * x + torch.cos(ph) * y)
    m = unit(torch.stack([sx, sy, torch.ones_like(sx)]))  # the frame's x and y axes are -x and -y
    om = (w * m).sum(0)
    wi = -w + 2.0 * m * om
    eta = 1.0 / 1.5

    def fresnel(c1):
        c2 = torch.sqrt((1.0 - eta * eta * (1.0 - c1 * c1)).clamp_min(0.0))
        rs, rp = (eta * c1 - c2) / (eta * c1 + c2), (c1 - eta * c2) / (c1 + eta * c2)
        return torch.where(c2 > 0, 0.5 * (rs * rs + rp * rp), torch.ones_like(c1))

    F = fresnel(om)
    refl = wi[2] > 0
    h = torch.where(refl, 1.0, -1.0) * unit(torch.where(refl, wi + w, eta * w + wi))

    def g1(v, m_):
        t2 = (1.0 - v[2] ** 2) / v[2] ** 2
        q = torch.sqrt(1.0 / (a * a * t2))
        bk = torch.where(q < 1.6, (3.535 * q + 2.181 * q * q) / (1.0 + 2.276 * q + 2.577 * q * q), torch.ones_like(q))
        return torch.where(v[2] * (v * m_).sum(0) <= 0, 0.0, torch.where(ggx, 2.0 / (1.0 + torch.sqrt(1.0 + a * a * t2)), bk))

    def ndf(z):
        t2 = (1.0 - z * z) / (z * z)
        gg = 1.0 / (math.pi * a * a * z ** 4 * (1.0 + t2 / (a * a)) ** 2)
        return torch.where(ggx, gg, torch.exp(-t2 / (a * a)) / (math.pi * a * a * z ** 4))

    Fh, G, D = fresnel((w * h).sum(0)), g1(w, h) * g1(wi, h), torch.where(h[2] > torch.where(ggx, 0.0, 1e-4), ndf(h[2]), 0.0)
    idm, odm = (w * h).sum(0).abs(), (wi * h).sum(0).abs()
    idn, odn = w[2].abs(), wi[2].abs()
    f = torch.where(refl, Fh * G * D / (4.0 * idn * odn), (1.0 - Fh) * G * D * idm * odm / (idn * odn) / (eta * idm + odm) ** 2)
    sz = torch.sqrt((1.0 - w[2] ** 2).clamp_min(0.0))
    b = w[2] / (sz * a)
    area = torch.where(ggx, 0.5 * (w[2] + torch.sqrt(w[2] ** 2 + sz * sz * a * a)),
                       0.5 * (torch.erf(b) + 1.0) * w[2] + 0.5 / math.sqrt(math.pi) * a * sz * torch.exp(-b * b))
    area = torch.where(w[2] > 0.9999, torch.ones_like(area), area)
    pdf = om.clamp_min(0.0) * ndf(m[2]) / area / (4.0 * om.abs())
    return {"wi": wi, "f": f, "pdf": pdf, "F": F}


def _rays_exact(case, seed):
    """The distance to the closest triangle, every ray against every triangle."""
    P = torch.from_numpy(_ray_scene(case, seed).flat_triangles()[0]).cuda().double().reshape(-1, 3, 3)
    o4, d4, _ = _rays(case, seed)
    o, d = o4[:, :3].double(), d4[:, :3].double()
    v0, e1, e2 = P[:, 0], P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    # with x = o - v0: t = -(x . n) / (d . n), u = -(x x d) . e2 / (d . n), v = (x x d) . e1 / (d . n)
    ray = torch.cat([torch.linalg.cross(o, d), d], 1)
    U = torch.cat([e2, torch.linalg.cross(v0, e2)], 1).T.contiguous()
    V = torch.cat([e1, torch.linalg.cross(v0, e1)], 1).T.contiguous()
    N, k, out = nrm.T.contiguous(), (v0 * nrm).sum(1), torch.empty(case["n"], dtype=torch.float64, device="cuda")
    step = max(1, (1 << 27) // len(P))
    for i in range(0, case["n"], step):
        dn = d[i:i + step] @ N
        r = ray[i:i + step]
        u = (r @ U).div_(dn).neg_()
        v = (r @ V).div_(dn)
        ok = (u >= 0) & (v >= 0) & (u.add_(v) <= 1)
        t = (k - o[i:i + step] @ N).div_(dn)
        ok &= t > 1e-4
        out[i:i + step] = t.masked_fill_(~ok, math.inf).amin(1)
    return torch.where(torch.isinf(out), -1.0, out)


def exact(case, seed):
    """BSDF queries and ray distances have a value in 64 bits.  A render is a Monte Carlo estimate whose
    sampled paths follow the 32-bit arithmetic (and a walk, a random path of the same kind), so those have none."""
    if case["kind"] == "bsdf":
        return _bsdf_exact(case, seed)
    if case["kind"] == "rays":
        if 20.0 * 4 ** case["subdiv"] * 1.25 * case["n"] > 6e10:
            return None  # above about 20 seconds
        return {"prim": None, "t": _rays_exact(case, seed), "bary": None, "hit": None}
    return None
