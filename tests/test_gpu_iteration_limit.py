"""A caller's max_iterations counts the iterations that a wave's rays need: one
per ray of the longest path while every path has a slot, and one more for each
time the pool is refilled. The smallest limit that suffices completes, one less
stops the render."""
import numpy as np
import pytest

from aurora_gb300 import api, scenes, types as T

pytestmark = pytest.mark.gpu


def _render(ctx, sc, p, pool, limit):
    b = api.Batch(ctx, [sc], [p], tuning=api.make_tuning(paths_in_flight=pool, samples_per_wave=1, max_iterations=limit))
    frame = b.render()[0].cpu().numpy()
    return frame, b.status()


def _suffices_exactly(ctx, sc, p, pool, limit, waves=1):
    want = sc.render(p).cpu().numpy()
    frame, iterations = _render(ctx, sc, p, pool, limit)
    assert iterations <= limit * waves and np.array_equal(frame, want)
    if limit > 1:
        with pytest.raises(api.AuroraError) as e:
            _render(ctx, sc, p, pool, limit - 1)
        assert e.value.status == 4


@pytest.mark.parametrize("mode", [T.MODE_PATH, T.MODE_PATH_MIS])
@pytest.mark.parametrize("depth", [0, 1, 4])
def test_one_pool_needs_an_iteration_per_ray_of_a_path(ctx, mode, depth):
    sc = api.Scene(ctx, scenes.cornell_emissive(area_light=True))
    p = T.render_params(64, 48, 2, depth, seed=3, mode=mode)
    _suffices_exactly(ctx, sc, p, 4096, depth + 1, waves=2)


@pytest.mark.parametrize("pool,pixels", [(1024, (64, 48)), (1024, (31, 33)), (2048, (64, 50)), (4096, (64, 64))])
def test_small_pools_of_paths_without_bounces(ctx, pool, pixels):
    sc = api.Scene(ctx, scenes.cornell())
    p = T.render_params(pixels[0], pixels[1], 1, 4, seed=3, mode=T.MODE_REFERENCE)
    _suffices_exactly(ctx, sc, p, pool, -(-pixels[0] * pixels[1] // pool))


@pytest.mark.parametrize("mode", [T.MODE_PATH, T.MODE_PATH_MIS])
def test_a_pool_smaller_than_the_frame(ctx, mode):
    sc = api.Scene(ctx, scenes.sphere_scene(3, min_tris=2000, max_tris=4000))
    p = T.render_params(96, 80, 1, 3, seed=5, mode=mode)
    _, needed = _render(ctx, sc, p, 1024, 100000)
    # a slot is handed back in the iteration its path ends in: the pool is full
    # until the last of the frame's rays (four a path at most) have started
    assert needed <= -(-4 * 96 * 80 // 1024) + 3
    _suffices_exactly(ctx, sc, p, 1024, needed)


def test_stepped_and_graph_renders_agree_with_a_limit(ctx):
    import torch
    sc = api.Scene(ctx, scenes.cornell_sphere(seed=2, slices=16, stacks=8))
    p = T.render_params(40, 30, 3, 4, seed=5, mode=T.MODE_PATH)
    for limit in (0, 50):
        b = api.Batch(ctx, [sc], [p], tuning=api.make_tuning(paths_in_flight=1024, max_iterations=limit))
        f = [torch.zeros((30, 40, 4), device="cuda")]
        b.profile(f)
        assert torch.equal(f[0], b.render()[0])
        b.status()
