"""scenes.sphere_scene: a scene for every limit on its triangles that a sphere
fits, also where the first sphere drawn is larger than the limit."""
import pytest

from aurora_gb300 import scenes


@pytest.mark.parametrize("max_tris", [80, 100, 500, 2000, 2600, 5000, 20000])
def test_every_seed_gives_a_scene_within_the_limit(max_tris):
    for seed in range(60):
        sd = scenes.sphere_scene(seed, min_tris=min(1000, max_tris), max_tris=max_tris)
        assert 12 <= sd.count <= max_tris


def test_a_limit_below_every_sphere_is_refused():
    with pytest.raises(ValueError):
        scenes.sphere_scene(0, min_tris=1, max_tris=79)
