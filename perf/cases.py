"""The workloads this library is timed on: what a renderer built on it asks for.

Each case is one pass through the public entry points (aurora_gb300.api, the
ctypes form of include/aurora_gb300.h) over inputs made from a seed:

  trace       closest hit or any hit for a buffer of rays, on the device or
              through host buffers, against a triangle soup or a small scene
  build       the per-frame rebuild of the acceleration structure: aur_nmh_build
              and aur_nmh_apply of the vertices and of the prim ids
  render      aur_render: one frame of one scene, every sample in one call
  batch       aur_batch_render: wavefront frames of several scenes (or one
              large scene) as one call
  adjoint     aur_render_adjoint: gradients for an image gradient
  filter      aur_filter_pixels of a finished frame

Scenes come from aurora_gb300.scenes, ray and soup distributions are those of
its random_soup() and microbench_rays().
"""
import ctypes
import math

import numpy as np
import torch

from aurora_gb300 import api, scenes
from aurora_gb300 import types as T

_ctx = None


def _context():
    """One library context per process, as a renderer keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = api.Context(0)
    _ctx.use_torch_stream()
    return _ctx


# ------------------------------------------------------------------- cases

def listed():
    return [
        # picking and probing rays in a tiny scene: a call is all latency
        {"name": "trace_closest_box_4k", "kind": "trace", "any": False, "host": False, "scene": "cornell", "tris": 34,
         "rays": "camera", "n": 4099},
        # the traversal microbench: half a camera's rays, half random ones, 1M triangles
        {"name": "trace_closest_soup_16m", "kind": "trace", "any": False, "host": False, "scene": "soup",
         "tris": 1000000, "rays": "mixed", "n": 1 << 24},
        # shadow rays from anywhere in the scene toward one area light
        {"name": "trace_any_soup_4m", "kind": "trace", "any": True, "host": False, "scene": "soup", "tris": 1000000,
         "rays": "light", "n": 4194301},
        # a caller whose rays and hits live in (pinned) host memory
        {"name": "trace_closest_host_6m", "kind": "trace", "any": False, "host": True, "scene": "soup",
         "tris": 300000, "rays": "mixed", "n": 6000000},
        # the per-frame rebuild of a deforming mesh: small and large
        {"name": "build_20k", "kind": "build", "tris": 20001},
        {"name": "build_1m", "kind": "build", "tris": 1000000},
        # a preview frame of a small scene, and the estimator with light sampling
        {"name": "render_box_256", "kind": "render", "scene": "cornell", "tris": 34, "mode": T.MODE_PATH, "width": 256,
         "height": 256, "spp": 16, "depth": 4},
        {"name": "render_mis_emissive_300", "kind": "render", "scene": "cornell_emissive_area", "tris": 49,
         "mode": T.MODE_PATH_MIS, "width": 301, "height": 233, "spp": 9, "depth": 3},
        # a dataset of scenes rendered as one batch, and one large landscape
        {"name": "batch_spheres_8", "kind": "batch", "scene": "spheres", "tris": 500000, "scenes": 8,
         "mode": T.MODE_PATH, "width": 512, "height": 512, "spp": 4, "depth": 6},
        {"name": "batch_terrain_2m", "kind": "batch", "scene": "terrain", "tris": 2 * 1023 * 1023, "scenes": 1,
         "mode": T.MODE_PATH, "width": 960, "height": 540, "spp": 2, "depth": 8},
        # inverse rendering: the gradient of one frame's loss
        {"name": "adjoint_sphere_256", "kind": "adjoint", "scene": "cornell_sphere", "tris": 4130, "mode": T.MODE_PATH,
         "width": 256, "height": 256, "spp": 16, "depth": 4},
        # the display filter of a 4K frame
        {"name": "filter_4k", "kind": "filter", "width": 3840, "height": 2160, "region": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "trace", "build", "render", "render", "batch", "adjoint", "filter"])
    if kind == "trace":
        return {"kind": kind, "any": rng.random() < 0.4, "host": rng.random() < 0.2, "scene": "soup",
                "tris": _log(rng, 34, 2000000), "rays": rng.choice(["camera", "random", "mixed", "light"]),
                "n": _log(rng, 1000, 1 << 23)}
    if kind == "build":
        return {"kind": kind, "tris": _log(rng, 300, 3000000)}
    if kind == "filter":
        return {"kind": kind, "width": _log(rng, 64, 3840), "height": _log(rng, 48, 2160), "region": rng.random() < 0.5}
    side = _log(rng, 64, 512)
    case = {"kind": kind, "width": side, "height": max(1, int(side * rng.uniform(0.5, 1.0))),
            "mode": rng.choice([T.MODE_REFERENCE, T.MODE_PATH, T.MODE_PATH, T.MODE_PATH_MIS]), "depth": rng.randint(1, 6)}
    if kind == "batch":
        case.update(scene="spheres", tris=_log(rng, 2000, 300000), scenes=rng.randint(1, 6), spp=_log(rng, 1, 6))
    else:
        case.update(scene=rng.choice(["cornell", "cornell_emissive_area", "cornell_sphere", "cornell_specular",
                                      "cornell_textured", "spheres"]), tris=_log(rng, 2000, 200000), spp=_log(rng, 1, 20))
        if kind == "adjoint" and case["scene"] == "cornell_textured":
            case["scene"] = "cornell_specular"
    return case


# ------------------------------------------------------------------ inputs

def _soup(n, g):
    """scenes.random_soup()'s distribution, made on the device: centroids
    U[0,1]^3, edges of LogNormal(-4, 0.5) length in uniform directions. The
    edge lengths grow as the count falls below 1M, so that a smaller soup
    still stops most rays."""
    c = torch.rand((n, 3), generator=g, device="cuda")
    length = torch.exp(torch.randn((n, 2, 1), generator=g, device="cuda") * 0.5 - 4.0) * (1e6 / max(n, 1)) ** 0.3
    d = torch.randn((n, 2, 3), generator=g, device="cuda")
    e = length * (d / d.norm(dim=2, keepdim=True))
    p1 = c - (e[:, 0] + e[:, 1]) / 3.0
    return torch.stack([p1, p1 + e[:, 0], p1 + e[:, 1]], 2).reshape(n, 9).contiguous()


def _box(g):
    """The Cornell box in world units that differ from seed to seed."""
    v = torch.from_numpy(scenes.cornell().vertices.copy()).cuda()
    scale = 0.8 + 0.4 * torch.rand(3, generator=g, device="cuda")
    return (v.reshape(-1, 3, 3) * scale[None, :, None]).reshape(-1, 9).contiguous()


def _camera_rays(n, g):
    """A pinhole before the unit cube looking +z, pixels in row order, the eye
    at another place for each seed."""
    side = max(1, int(math.sqrt(n)))
    k = torch.arange(n, device="cuda")
    px = ((k % side) + 0.5) / side - 0.5
    py = ((k // side) % side + 0.5) / side - 0.5
    eye = torch.tensor([0.5, 0.5, -1.0], device="cuda") + 0.1 * (torch.rand(3, generator=g, device="cuda") - 0.5)
    d = torch.stack([px, py, torch.ones_like(px)], 1)
    return eye.expand(n, 3), d / d.norm(dim=1, keepdim=True), torch.full((n,), 1.0e6, device="cuda")


def _random_rays(n, g):
    o = torch.rand((n, 3), generator=g, device="cuda")
    d = torch.randn((n, 3), generator=g, device="cuda")
    return o, d / d.norm(dim=1, keepdim=True), torch.full((n,), 1.0e6, device="cuda")


def _light_rays(n, g):
    """Segments from points in the cube to points of a square light above it."""
    o = torch.rand((n, 3), generator=g, device="cuda")
    q = torch.rand((n, 3), generator=g, device="cuda") * torch.tensor([0.5, 0.0, 0.5], device="cuda")
    d = q + torch.tensor([0.25, 1.6, 0.25], device="cuda") - o
    t = d.norm(dim=1)
    return o, d / t[:, None], t


def _rays(kind, n, g):
    if kind == "mixed":
        a, b = _camera_rays(n // 2, g), _random_rays(n - n // 2, g)
        o, d, t = (torch.cat([x, y]) for x, y in zip(a, b))
    else:
        o, d, t = {"camera": _camera_rays, "random": _random_rays, "light": _light_rays}[kind](n, g)
    r = torch.zeros((n, 8), dtype=torch.float32, device="cuda")
    r[:, 0:3], r[:, 3], r[:, 4:7] = o, t, d
    return r


def _trace_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    verts = _box(g) if case["scene"] == "cornell" else _soup(case["tris"], g)
    rays = _rays(case["rays"], case["n"], g)
    if case["scene"] == "cornell":
        # the box opens toward +z: its camera stands there and looks back
        rays[:, 2] = 2.3 + 0.1 * torch.rand(1, generator=g, device="cuda")
        rays[:, 6] = -rays[:, 6]
    return verts, rays


def _specular(seed):
    sd = scenes.cornell()
    sh = np.concatenate([sd.shaders, np.stack([T.lambert(scenes.WHITE), T.lambert(scenes.WHITE)])])
    sh["reflectivity"][3] = 0.8
    sh["translucence"][4], sh["reflectivity"][4], sh["refractive_index"][4] = 0.8, 0.1, 1.5
    ids = sd.shader_ids.copy()
    ids[10:22], ids[22:34] = 4, 5     # a mirror block and a glass block
    return scenes.SceneData("cornell_specular", sd.vertices, sd.normals, ids, sh, sd.lights, sd.camera)


def _scene_data(case, seed, i=0):
    name = case["scene"]
    if name == "spheres":
        return scenes.sphere_scene(seed * 64 + i, min_tris=min(1000, case["tris"]), max_tris=case["tris"])
    if name == "terrain":
        return scenes.terrain(res=int(round(math.sqrt(case["tris"] / 2.0))) + 1, seed=seed)
    sd = {"cornell": scenes.cornell, "cornell_emissive_area": lambda: scenes.cornell_emissive(area_light=True),
          "cornell_sphere": lambda: scenes.cornell_sphere(seed), "cornell_specular": lambda: _specular(seed),
          "cornell_textured": lambda: scenes.cornell_textured(seed)}[name]()
    rng = np.random.default_rng(seed)
    cam = sd.camera.copy()      # the eye at another place for each seed
    cam["position"] = cam["position"] + rng.uniform(-0.05, 0.05, 3).astype(np.float32)
    sd.camera = cam
    return sd


def _params(case, seed, i=0):
    return T.render_params(case["width"], case["height"], case["spp"], case["depth"], seed=seed, mode=case["mode"],
                           scene_id=i)


def _region(case):
    if not case["region"]:
        return None
    w, h = case["width"], case["height"]
    return (w // 5, w - 1 - w // 7, h // 6, h - 1 - h // 9)


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    s = {"case": case, "ctx": ctx}
    if kind == "trace":
        verts, rays = _trace_inputs(case, seed)
        s["nmh"] = api.Nmh(ctx, verts)
        if case["host"]:
            s["rays"] = rays.cpu().pin_memory()
            s["hits"] = torch.empty((case["n"], 4), dtype=torch.float32).pin_memory()
        else:
            s["rays"] = rays
    elif kind == "build":
        g = torch.Generator(device="cuda").manual_seed(seed)
        s["verts"] = _soup(case["tris"], g)
        s["ids"] = torch.arange(case["tris"], dtype=torch.int32, device="cuda")
    elif kind == "filter":
        g = torch.Generator(device="cuda").manual_seed(seed)
        # radiance spans several orders of magnitude; alpha is the coverage
        img = torch.exp(torch.randn((case["height"], case["width"], 4), generator=g, device="cuda"))
        img[..., 3] = torch.rand((case["height"], case["width"]), generator=g, device="cuda")
        s["img"], s["out"] = img, torch.zeros_like(img)
    else:
        many = case.get("scenes", 1)
        s["scenes"] = []
        for i in range(many):
            sd = _scene_data(case, seed, i)
            sc = api.Scene(ctx, sd)
            if hasattr(sd, "textures"):
                sc.set_textures(sd.texcoords, sd.textures)
            s["scenes"].append(sc)
        s["params"] = [_params(case, seed, i) for i in range(many)]
        if kind == "batch":
            s["batch"] = api.Batch(ctx, s["scenes"], s["params"], tuning=api.make_tuning(paths_in_flight=1 << 22))
        if kind == "adjoint":
            g = torch.Generator(device="cuda").manual_seed(seed)
            # dLoss/dimage of a squared difference: both signs, every pixel
            s["d_image"] = torch.randn((case["height"], case["width"], 4), generator=g, device="cuda")
    return s


# -------------------------------------------------------------------- pass

def _hits(h):
    """(t, u, v) and the prim ids of an aur_hit buffer, as views."""
    return [h[:, :3], h.view(torch.int32)[:, 3]]


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "trace":
        if case["host"]:
            if case["any"]:
                occ = state["hits"].view(torch.int32).reshape(-1)[:case["n"]]
                return [api.trace_any_host(ctx, state["nmh"], state["rays"], occ)]
            return _hits(api.trace_closest_host(ctx, state["nmh"], state["rays"], state["hits"]))
        if case["any"]:
            return [api.trace_any(ctx, state["nmh"], state["rays"])]
        return _hits(api.trace_closest(ctx, state["nmh"], state["rays"]))
    if kind == "build":
        nmh = api.Nmh(ctx, state["verts"])
        count, _ = nmh.info()
        verts = torch.empty((count, 9), dtype=torch.float32, device="cuda")
        ids = torch.empty((count,), dtype=torch.int32, device="cuda")
        for src, size, dst in ((state["verts"], 36, verts), (state["ids"], 4, ids)):
            api.check(api.lib().aur_nmh_apply(ctx.handle, nmh.handle, ctypes.c_void_p(src.data_ptr()), size,
                                              ctypes.c_void_p(dst.data_ptr())))
        nmh.close()
        return [verts, ids]
    if kind == "filter":
        api.filter_pixels(ctx, case["width"], case["height"], state["img"], state["out"], region=_region(case))
        return [state["out"]]
    if kind == "render":
        return [state["scenes"][0].render(state["params"][0])]
    if kind == "batch":
        return state["batch"].render()
    return list(state["scenes"][0].adjoint(state["params"][0], state["d_image"], emission=True))


# -------------------------------------------------------------- accounting

# what one ray cannot do without: a binary descent of the triangles (two box
# tests of 12 operations a level) and one triangle test (about 50 operations)
def _ray_flops(tris):
    return 24 * max(1.0, math.log2(max(2, tris))) + 50


def work(case):
    kind = case["kind"]
    if kind == "trace":
        n, tris = case["n"], case["tris"]
        return {"bytes": n * (28 + (4 if case["any"] else 16)) + 36 * tris, "flops": n * _ray_flops(tris)}
    if kind == "build":
        n = case["tris"] + case["tris"] % 2
        # vertices in; permuted vertices and ids out; the 128-byte node records, one per two triangles
        return {"bytes": n * (36 + 36 + 4 + 64), "flops": n * 2 * max(1.0, math.log2(max(2, n)))}
    if kind == "filter":
        r = _region(case) or (0, case["width"] - 1, 0, case["height"] - 1)
        px = (r[1] - r[0] + 1) * (r[3] - r[2] + 1)
        return {"bytes": 32 * px, "flops": 17 * 4 * px}
    scenes_ = case.get("scenes", 1)
    px = case["width"] * case["height"] * scenes_
    lights = 16 if case["scene"] == "terrain" else 1
    hits = 1 if case["mode"] == T.MODE_REFERENCE else case["depth"] + 1
    rays = px * case["spp"] * hits * (1 + lights)
    tris = {"cornell": 34, "cornell_emissive_area": 49, "cornell_sphere": 4130, "cornell_specular": 34,
            "cornell_textured": 34}.get(case["scene"], case["tris"])
    return {"bytes": 16 * px + 74 * tris * scenes_, "flops": rays * _ray_flops(tris)}


# ------------------------------------------------------------ 64-bit values

def _exact_filter(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    img = torch.exp(torch.randn((case["height"], case["width"], 4), generator=g, device="cuda"))
    img[..., 3] = torch.rand((case["height"], case["width"]), generator=g, device="cuda")
    img = img.double()
    l, r, b, t = _region(case) or (0, case["width"] - 1, 0, case["height"] - 1)
    win = img[b:t + 1, l:r + 1]
    xs = torch.arange(r - l + 1, device="cuda")
    ys = torch.arange(t - b + 1, device="cuda")
    acc = torch.zeros_like(win)
    for dy, wy in ((-1, 0.25), (0, 0.5), (1, 0.25)):
        row = win[(ys + dy).clamp(0, t - b)]
        for dx, wx in ((-1, 0.25), (0, 0.5), (1, 0.25)):
            acc += wy * wx * row[:, (xs + dx).clamp(0, r - l)]
    out = torch.zeros_like(img)
    out[b:t + 1, l:r + 1] = acc
    return [out]


def _exact_trace(case, seed):
    """The nearest front-facing triangle of each ray, every pair tested (the
    distance and barycentrics; the prim ids are whole numbers)."""
    verts, rays = _trace_inputs(case, seed)
    v = verts.double().reshape(-1, 3, 3)          # triangle, axis, corner
    p1, e1, e2 = v[:, :, 0], v[:, :, 1] - v[:, :, 0], v[:, :, 2] - v[:, :, 0]
    out = []
    for r in rays.double().split(max(1, (1 << 22) // verts.shape[0])):
        o, d, tmax = r[:, None, 0:3], r[:, None, 4:7], r[:, 3]
        P = torch.linalg.cross(d, e2[None])
        det = (e1[None] * P).sum(2)
        q = o - p1[None]
        u = (q * P).sum(2) / det
        Q = torch.linalg.cross(q, e1[None].expand_as(q))
        w = (d * Q).sum(2) / det
        t = (e2[None] * Q).sum(2) / det
        ok = (det >= 1e-7) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 1e-7) & (t < tmax[:, None])
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        best, k = t.min(1)
        hit = torch.isfinite(best)
        k = k[:, None]
        zero = torch.zeros_like(best)
        out.append(torch.stack([torch.where(hit, best, tmax), torch.where(hit, u.gather(1, k)[:, 0], zero),
                                torch.where(hit, w.gather(1, k)[:, 0], zero)], 1))
    return [torch.cat(out), None]


def exact(case, seed):
    if case["kind"] == "filter":
        return _exact_filter(case, seed)
    if case["kind"] == "trace":
        if case["any"]:
            return None                         # prim ids only
        # every ray against every triangle: up to 2^31 pairs take a few seconds
        return _exact_trace(case, seed) if case["n"] * case["tris"] <= 1 << 31 else None
    # builds give vertices as they were and prim ids. Frames and gradients are
    # Monte-Carlo sums whose every term hangs on which triangle a ray meets
    # and which light it sees, decided in 32 bits from 32-bit random numbers:
    # they have no 64-bit value.
    return None
