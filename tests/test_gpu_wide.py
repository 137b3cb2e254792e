"""The trace kernels over every route a launch can take (a few triangles with
no tree, a launch that fits the GPU at once, a larger one; packets, one ray
per lane, deferred chunks) against the oracle, at the sizes where a route or a
partial chunk begins and ends. Results are equal bit for bit."""
import numpy as np
import pytest

import oracle
from aurora_gb300 import api, scenes, types as T
from helpers import hits_equal

pytestmark = pytest.mark.gpu


def _rays(kind, n, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros(n, T.ray_dtype)
    r["tmax"] = 1e6
    if kind == "pinhole":           # narrow, wide and mixed-octant chunks of one eye
        side = max(1, int(np.sqrt(n)))
        k = np.arange(n)
        d = np.stack([(k % side + 0.5) / side - 0.5, (k // side + 0.5) / side - 0.5, np.ones(n)], 1)
        o = np.tile([0.5, 0.5, -1.0], (n, 1))
    else:
        d = rng.normal(size=(n, 3))
        o = rng.random((n, 3))
        r["tmax"][::5] = 0.3
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r["ox"], r["oy"], r["oz"] = o.astype(np.float32).T
    r["dx"], r["dy"], r["dz"] = d.astype(np.float32).T
    return r


def _soup(n, seed):
    rng = np.random.default_rng(seed)
    size = 0.9 * n ** (-1.0 / 3.0)
    c = rng.random((n, 3, 1))
    return (c + rng.normal(size=(n, 3, 3)) * size * 0.5).astype(np.float32).reshape(-1, 9)


@pytest.mark.parametrize("kind", ["pinhole", "random"])
@pytest.mark.parametrize("n_tris,n_rays", [(1, 33), (2, 1), (3, 31), (33, 4099), (63, 9729), (64, 9728), (64, 130001),
                                           (65, 4099), (66, 32), (129, 1000), (5000, 40000), (300, 116736),
                                           (300, 116737), (5000, 150013)])
def test_every_route_matches_oracle(ctx, kind, n_tris, n_rays):
    import torch
    V = _soup(n_tris, n_tris)
    nmh = api.Nmh(ctx, torch.from_numpy(V.reshape(-1)).cuda(), count=n_tris)
    perm, verts = nmh.export()
    rays = _rays(kind, n_rays, n_tris + n_rays)
    hits = api.hits_to_numpy(api.trace_closest(ctx, nmh, api.rays_tensor(rays)))
    occ = api.trace_any(ctx, nmh, api.rays_tensor(rays)).cpu().numpy().view(np.uint32)
    ohits, _, _ = oracle.trace_closest(verts, perm, rays)
    oocc, _, _ = oracle.trace_any(verts, perm, rays)
    assert hits_equal(hits, ohits)
    assert np.array_equal(occ, oocc)
    assert n_tris < 60 or n_rays < 100 or (hits["prim"] != T.NO_HIT).any()
