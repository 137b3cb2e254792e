"""Rays whose whole direction vector is short (aur_ray does not ask for unit
directions): the box tests of the treelets and the filter in front of a few
triangles must not bend them. The treelets' host build (tests/wide_model.cpp)
against the oracle's walk without boxes, bit for bit, with triangles large
enough that Moller-Trumbore's det >= 1e-7 can be met at all."""
import numpy as np
import pytest

from test_wide_model import _check, _rays, model  # noqa: F401  (model: the module's fixture)


def _short_rays(n_tris, length, seed):
    """Triangles and rays aimed at them; among the rays some with one zero
    component and some parallel to an axis, along which a bent ray goes
    furthest astray."""
    rng = np.random.default_rng(seed)
    size = max(1.0, 3.0 * np.sqrt(1e-7 / length))
    V = ((rng.random((n_tris, 3, 1)) * 2.0 + rng.normal(size=(n_tris, 3, 3)) * 0.5) * size).astype(np.float32)
    n = 3000
    P = V[rng.integers(0, n_tris, n)].astype(np.float64)          # triangle, axis, corner
    a, b = rng.random((2, n))
    b *= 1.0 - a
    o = rng.random((n, 3)) * 2.0 * size
    d = P[:, :, 0] + a[:, None] * (P[:, :, 1] - P[:, :, 0]) + b[:, None] * (P[:, :, 2] - P[:, :, 0]) - o
    d[:600, rng.integers(0, 3)] = 0.0
    d[600:1200] = 0.0
    d[np.arange(600, 1200), rng.integers(0, 3, 600)] = rng.choice([-1.0, 1.0], 600)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return V.reshape(-1, 9), _rays(o, d * length, 1.0e38)


@pytest.mark.parametrize("exponent", [-6, -8, -9, -11, -12, -13, -15, -18, -19, -20, -21, -22, -23, -24, -26, -28])
@pytest.mark.parametrize("n_tris", [40, 400])
def test_short_directions_match_the_walk_without_boxes(model, n_tris, exponent):  # noqa: F811
    V, rays = _short_rays(n_tris, 10.0 ** exponent, -exponent)
    hits, _ = _check(model, V, rays)
    assert (hits["prim"] != 0xFFFFFFFF).any()


def test_mixed_lengths_and_zero_directions(model):  # noqa: F811
    """Lengths from 1 to below the smallest normal float in one launch, some
    rays without any direction (these hit nothing)."""
    V, rays = _short_rays(300, 1e-13, 7)
    rng = np.random.default_rng(8)
    scale = 10.0 ** rng.uniform(-45.0, 13.0, len(rays))
    for f in ("dx", "dy", "dz"):
        rays[f] = (rays[f].astype(np.float64) * scale).astype(np.float32)
        rays[f][::50] = 0.0
    hits, _ = _check(model, V, rays)
    assert (hits["prim"] != 0xFFFFFFFF).sum() > 300 and np.all(hits["prim"][::50] == 0xFFFFFFFF)
