"""The adjoint's replay without a ray stack (scenes with no specular shader)
against its replay with one: a specular shader that no triangle uses selects
the latter, so both must give the same gradients up to the order of the sums."""
import numpy as np
import pytest

from aurora_gb300 import api, scenes, types as T

pytestmark = pytest.mark.gpu

W, H, SPP = 37, 21, 4


def _scene(kind):
    sd = {"tiny": scenes.cornell, "tiny_emissive": lambda: scenes.cornell_emissive(area_light=True),
          "tree_many": lambda: scenes.cornell_sphere(seed=2, slices=16, stacks=8),
          "tree_few": lambda: scenes.sphere_scene(4, min_tris=2000, max_tris=4000)}[kind]()
    sd.shaders = np.concatenate([sd.shaders, np.stack([T.lambert((0.5, 0.5, 0.5))])])
    return sd


@pytest.mark.parametrize("mode", [T.MODE_REFERENCE, T.MODE_PATH, T.MODE_PATH_MIS])
@pytest.mark.parametrize("depth", [0, 1, 5, 16])
@pytest.mark.parametrize("kind", ["tiny", "tiny_emissive", "tree_many", "tree_few"])
def test_replay_without_a_stack_equals_the_one_with(kind, depth, mode):
    import torch
    ctx = api.Context(0)
    sd = _scene(kind)
    sc = api.Scene(ctx, sd)
    p = T.render_params(W, H, SPP, depth, seed=9, mode=mode)
    ones = torch.ones((H, W, 4), dtype=torch.float32, device="cuda")
    plain = [g.cpu().numpy().astype(np.float64) for g in sc.adjoint(p, ones, emission=True)]
    sh = sd.shaders.copy()
    sh["reflectivity"][-1] = 0.5
    sc.set_shaders(sh)
    stack = [g.cpu().numpy().astype(np.float64) for g in sc.adjoint(p, ones, emission=True)]
    # every term is >= 0 and the same on both sides; a sum of n such floats is
    # off by at most n roundings, whatever its order (two terms a vertex)
    n = 2 * W * H * SPP * (depth + 1)
    for a, b in zip(plain, stack):
        assert np.all(a >= 0.0) and np.isfinite(a).all()
        np.testing.assert_allclose(a, b, rtol=2.0 * n * 2.0 ** -24, atol=0.0)
    assert plain[1].max() > 0.0 or len(sd.lights) == 0
