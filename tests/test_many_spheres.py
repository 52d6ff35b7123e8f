"""Worlds of many spheres against the oracle, bit for bit: the first GJK pass lets pairs with a sphere run on
where a warp holds several of them. From half of the bodies on, hulls of more than eight points among the
others; steps of more than 2,432 candidates (below, every pair has a warp)."""
import numpy as np
import pytest

from test_narrow_paths import _compare, _hull_scene

pytestmark = pytest.mark.gpu


def _with_spheres(sc, n, seed, radius):
    """The scene's cubes, and n spheres: resting on the ground beside them, the last few falling."""
    from nans_projekat_gb300 import scenes
    rng = np.random.default_rng(seed)
    r = radius * rng.uniform(0.8, 1.2, n)
    up = np.where(np.arange(n) < n - n // 4, 0.98 * r, 3.0 + rng.uniform(0.0, 2.0, n))
    pos = np.stack([-8.0 - 1.7 * np.arange(n), up, rng.uniform(-0.6, 0.6, n)], axis=1)
    sp = scenes._spheres(pos, r, 1.0 + r, 0.1, vel=rng.normal(0.0, 1.0, (n, 3)))
    return scenes.Scene(sc.cubes, sp, scenes.ground(200.0), cube_scale=sc.cube_scale, hull_npts=sc.hull_npts,
                        hull_pts=sc.hull_pts)


@pytest.mark.parametrize("kind,n_scenes,boxes,spheres", [
    ("stack", 1, 2, 8), ("stack", 180, 1, 20), ("stack", 1500, 1, 1), ("stack", 300, 6, 6), ("stack", 300, 7, 6),
    ("hulls", 200, 14, 16), ("hulls", 160, 14, 40)])
def test_many_spheres(oracle_lib, kind, n_scenes, boxes, spheres):
    from nans_projekat_gb300 import scenes
    batch = []
    seeds = [s for s in range(2 * n_scenes) if (scenes.mixed_scene(scenes.SplitMix64(s), 14).hull_npts > 0).any()]
    for i in range(n_scenes):
        sc = scenes.stack_scene_random(scenes.SplitMix64(100 + i), boxes + 1) if kind == "stack" else \
            _hull_scene(scenes, 9 + i % 6, seeds[i])
        batch.append(_with_spheres(sc, spheres, i, 0.45))
    _compare(batch, 25, lambda w, n: w.batch_step(np.float32(1.0 / 60.0), n, 5))
