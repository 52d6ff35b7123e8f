"""nans_launches_per_step counts the kernels that a step launches: by the size of the world (the pair
tier alone for few pairs, the long GJK runs by a kernel of their own for many bodies) and by the cull's
form (the tiles and the placement, or the placement alone)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DT = np.float32(1.0 / 60.0)


def _stacks(n, bodies):
    from nans_projekat_gb300 import scenes
    some = scenes.stack_batch(min(n, 50), seed=8, lo=bodies, hi=bodies)
    return (some * (n // len(some) + 1))[:n]


@pytest.mark.parametrize("scenes_bodies,flags,tiles,launches", [
    ((1, 9), {}, 1, 9),                       # sweep, 2 cull, pair tier, 3 EPA tiers, 2 solve
    ((1, 9), dict(all_pairs=True), 1, 8),     # the cull's mask in its placement
    ((1, 9), {}, 0, 8),
    ((1, 9), dict(gjk_warp=True), 1, 12),
    ((300, 40), {}, 1, 12),                   # GJK, pair tier twice and per-thread EPA
    ((300, 40), {}, 0, 11),
    ((2100, 40), {}, 1, 13),                  # and the long GJK runs
])
def test_kernels_of_a_staged_step(scenes_bodies, flags, tiles, launches):
    from nans_projekat_gb300 import lib
    w = lib.World(**flags)
    w.upload_batch(_stacks(*scenes_bodies))
    t = w.tuning()
    w.set_tuning(t["gjk_blocks_per_sm"], t["solve_threads"], t["solve_threads_late"], cull_tiles=tiles)
    w.step(DT, 1)
    assert w.launches_per_step() == (launches, launches)
    w.close()
