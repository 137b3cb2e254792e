"""Hard inputs through each route of a trace. Launches of more rays than the GPU
holds at once hand their mixed chunks to the refilling one-ray-per-lane kernel;
smaller ones trace them on the spot, coherent chunks go as packets. The same
rays, in an order that asks for the route, against the oracle, bit for bit:
ties, NaN and infinities, zero components of both signs, segments that end
before Epsilon, grazing rays far from the origin, directions from 1e-21 to 1,
and a last chunk that is not full."""
import numpy as np
import pytest

import oracle
from aurora_gb300 import api, scenes, types as T
from helpers import hits_equal
from test_short_directions import _short_rays

pytestmark = pytest.mark.gpu

RAYS_PER_SM = 6 * 128      # up to this many rays per SM, mixed chunks stay in the first launch


def _rays(o, d, tmax=1.0e6):
    r = np.zeros(len(o), T.ray_dtype)
    r["ox"], r["oy"], r["oz"] = np.asarray(o, np.float32).T
    r["dx"], r["dy"], r["dz"] = np.asarray(d, np.float32).T
    r["tmax"] = tmax
    return r


def _unit(d):
    return d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-30)


def _ties():
    rng = np.random.default_rng(1)
    V = scenes.random_soup(4000, seed=5)
    V[3000:3300] = V[100:400]
    V[3300:3600] = V[100:400]
    c = V[100:400].reshape(-1, 3, 3).mean(2)[rng.integers(0, 300, 4000)]
    o = c + rng.normal(size=c.shape) * 0.2
    r = _rays(o, _unit(c - o))
    r["tmax"][::7] = np.linalg.norm(c - o, axis=1)[::7]       # ending at the copies
    return V, r


def _non_finite():
    V = scenes.random_soup(20000, seed=8)
    r = scenes.microbench_rays(8192, seed=9)[4096:].copy()    # its random half
    values = (np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-42, 1e30)
    for j in range(0, 4096, 3):
        r[("ox", "oy", "oz", "dx", "dy", "dz", "tmax")[j // 3 % 7]][j] = values[j // 21 % 7]
    return V, r


def _lattice():
    rng = np.random.default_rng(3)
    n, m = 6000, 6000
    c = rng.integers(0, 32, size=(n, 3)).astype(np.float32) / 32.0
    e = rng.integers(1, 4, size=(n, 2)).astype(np.float32) / 128.0
    flat = rng.integers(0, 3, size=n)
    k = np.arange(n)
    p2, p3 = c.copy(), c.copy()
    p2[k, (flat + 1) % 3] += e[:, 0]
    p3[k, (flat + 2) % 3] += e[:, 1]
    swap = rng.random(n) < 0.5
    p2[swap], p3[swap] = p3[swap], p2[swap].copy()
    o = rng.integers(-4, 36, size=(m, 3)).astype(np.float32) / 32.0
    o[: m // 4] = c[rng.integers(0, n, m // 4)]
    d = np.zeros((m, 3), np.float32)
    d[np.arange(m), rng.integers(0, 3, m)] = rng.choice([-1.0, 1.0], m)
    d[d == 0] = np.where(rng.random((d == 0).sum()) < 0.5, 0.0, -0.0)
    d[m // 2:] = _unit(rng.normal(size=(m - m // 2, 3)))
    d[3 * m // 4:, 1] = -0.0
    return scenes.tris_to_soa(c, p2, p3), _rays(o, d)


def _short_segments():
    V = scenes.random_soup(30000, seed=4)
    r = scenes.microbench_rays(8192, seed=10)[4096:].copy()
    rng = np.random.default_rng(4)
    r["tmax"] = rng.choice(np.array([1e-9, 1e-7, 2e-7, 0.0, -1.0, 0.01, 0.3, 1e6], np.float32), 4096)
    return V, r


def _grazing():
    rng = np.random.default_rng(5)
    V = scenes.random_soup(20000, seed=7).reshape(-1, 3, 3)
    V = (V + np.array([1000.0, -2000.0, 500.0], np.float32)[:, None]).astype(np.float32)
    m = 4096
    t = V[rng.integers(0, len(V), m)].astype(np.float64)
    v1, e1, e2 = t[:, :, 0], t[:, :, 1] - t[:, :, 0], t[:, :, 2] - t[:, :, 0]
    a, b = rng.random((2, m, 1))
    b *= 1.0 - a
    d = _unit(_unit(e1) + rng.uniform(1e-4, 0.05, (m, 1)) * _unit(np.cross(e2, e1)))
    return V.reshape(-1, 9), _rays(v1 + a * e1 + b * e2 - d * rng.uniform(0.001, 3.0, (m, 1)), d)


def _short_directions():
    V, r = _short_rays(400, 1e-13, 11)
    rng = np.random.default_rng(11)
    scale = 10.0 ** rng.uniform(-8.0, 13.0, len(r))
    for f in ("dx", "dy", "dz"):
        r[f] = (r[f].astype(np.float64) * scale).astype(np.float32)
        r[f][::40] = 0.0
    return V, r


def _few_triangles():
    V, r = _short_rays(60, 1e-13, 12)
    rng = np.random.default_rng(12)
    scale = 10.0 ** rng.uniform(-12.0, 13.0, len(r))
    for f in ("dx", "dy", "dz"):
        r[f] = (r[f].astype(np.float64) * scale).astype(np.float32)
    return V, r


INPUTS = {"ties": _ties, "non_finite": _non_finite, "lattice": _lattice, "short_segments": _short_segments,
          "grazing": _grazing, "short_directions": _short_directions, "few_triangles": _few_triangles}


@pytest.mark.parametrize("name", sorted(INPUTS))
@pytest.mark.parametrize("route", ["deferred", "on_the_spot", "packets", "host"])
def test_hard_inputs(ctx, name, route):
    import torch
    V, base = INPUTS[name]()
    V = np.ascontiguousarray(V, np.float32)
    nmh = api.Nmh(ctx, torch.from_numpy(V.reshape(-1)).cuda(), count=V.shape[0])
    perm, verts = nmh.export()
    rng = np.random.default_rng(17)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if route in ("deferred", "host"):
        n = sms * RAYS_PER_SM + 32 * 200 + 13
        pick = rng.integers(0, len(base), n)
    elif route == "on_the_spot":
        n = 32 * 120 + 7
        pick = rng.integers(0, len(base), n)
    else:                           # each ray 32 times over: one octant, one origin
        pick = np.repeat(rng.integers(0, len(base), sms * RAYS_PER_SM // 32 + 50), 32)[:-11]
        n = len(pick)
    # no chunk of the shuffled rays is of one octant: the first two of each differ
    octant = (base["dx"] < 0) * 1 + (base["dy"] < 0) * 2 + (base["dz"] < 0) * 4
    if route != "packets":
        pick[0::32] = rng.choice(np.flatnonzero(octant == 0), len(pick[0::32]))
        pick[1::32] = rng.choice(np.flatnonzero(octant == 7), len(pick[1::32]))
    rays = np.ascontiguousarray(base[pick])
    ohits, _, _ = oracle.trace_closest(verts, perm, base)
    oocc, _, _ = oracle.trace_any(verts, perm, base)
    if route == "host":
        hits, occ = np.zeros(n, T.hit_dtype), np.zeros(n, np.uint32)
        api.trace_closest_host(ctx, nmh, rays, hits)
        api.trace_any_host(ctx, nmh, rays, occ)
    else:
        rd = api.rays_tensor(rays)
        hits = api.hits_to_numpy(api.trace_closest(ctx, nmh, rd))
        if V.shape[0] > 64:         # fewer triangles have one route
            assert api.trace_deferred(ctx) == (0 if route == "packets" else (n + 31) // 32)
        occ = api.trace_any(ctx, nmh, rd).cpu().numpy().view(np.uint32)
    assert hits_equal(hits, ohits[pick])
    assert np.array_equal(occ, oocc[pick])
    assert (hits["prim"] != T.NO_HIT).any()
