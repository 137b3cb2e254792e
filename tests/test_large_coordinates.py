"""Axis-parallel rays in soups whose coordinates are large (1e8 to 1e16): the
products of a coordinate with the reciprocal of a zero component overflow, and
no box test may drop a triangle for it. The treelets' host build and the
node-by-node walk behind its checks against the oracle, bit for bit."""
import numpy as np
import pytest

from test_wide_model import _check, _rays, model  # noqa: F401  (model: the module's fixture)


@pytest.mark.parametrize("shift", [0.0, 1000.0])
@pytest.mark.parametrize("scale", [1.0, 1e8, 1e9, 1e12, 1e16])
@pytest.mark.parametrize("n_tris", [40, 1500])
def test_axis_parallel_rays_far_out(model, n_tris, scale, shift):  # noqa: F811
    rng = np.random.default_rng(n_tris)
    V = ((rng.random((n_tris, 3, 1)) + shift + rng.normal(size=(n_tris, 3, 3)) * 0.1) * scale).astype(np.float32)
    n = 3000
    P = V[rng.integers(0, n_tris, n)].astype(np.float64)
    a, b = rng.random((2, n, 1))
    b *= 1.0 - a
    target = P[:, :, 0] + a * (P[:, :, 1] - P[:, :, 0]) + b * (P[:, :, 2] - P[:, :, 0])
    d = np.zeros((n, 3))
    d[np.arange(n), rng.integers(0, 3, n)] = rng.choice([-1.0, 1.0], n)
    d[2000:, rng.integers(0, 3)] = 0.3                    # one component left at zero
    d[d == 0] = np.where(rng.random((d == 0).sum()) < 0.5, 0.0, -0.0)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = _rays(target - d * scale * rng.random((n, 1)) * rng.choice([1.0, 100.0], (n, 1)), d, 3.0e38)
    rays["tmax"][::3] = np.inf
    hits, _ = _check(model, V.reshape(-1, 9), rays)
    assert scale > 1e12 or (hits["prim"] != 0xFFFFFFFF).any()    # beyond, Moller-Trumbore itself overflows
