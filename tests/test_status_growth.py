"""The status bits of a call outlive a growth of its candidate buffers: a step whose grid-wide EPA tier
gave up on a pair is reported although a later step of the same call was put back and run again with
larger buffers."""
import numpy as np
import pytest

from helpers import GOLDEN_CASES, load_golden

pytestmark = pytest.mark.gpu


def _meeting_scene(n, step):
    """n heavy unit boxes that move 12 m a step towards one point: far apart before step `step`, on top of
    each other in it."""
    from nans_projekat_gb300 import scenes
    rng = np.random.default_rng(5)
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = 12.0 * (step - 1)
    pos = r * d + np.array([0.0, 2.0 * r + 100.0, 0.0])
    mass = rng.uniform(500.0, 2000.0, n)
    cubes = scenes._cubes(pos, None, mass, mass / 6.0, vel=-12.0 * 60.0 * d)
    return scenes.Scene(cubes, scenes._spheres(np.zeros((0, 3)), 0.5, np.zeros(0), np.zeros(0)), scenes.ground(60.0))


def _first_giant_step(lib):
    """The golden scene, and its step, whose EPA reaches the grid-wide tier first."""
    best = None
    for case in [c for c in GOLDEN_CASES if "bigepa" in c or "emptied" in c]:
        scene, meta, _, _ = load_golden(case)
        if not scene.rebuild_models:
            continue
        w = lib.World(giant_tier_only=True)
        w.upload(scene)
        last = meta["nsteps"] if best is None else min(meta["nsteps"], best[1] - 1)
        for k in range(1, last + 1):
            w.step(np.float32(scene.constants.dt), 1)
            if w.epa_stats()["giant_tier"]:
                best = (scene, k)
                break
        w.close()
    return best


@pytest.mark.parametrize("steps", ["graph", "eager"])
def test_timeout_before_a_growth_is_reported(steps):
    from nans_projekat_gb300 import lib
    scene, k = _first_giant_step(lib)
    dt = np.float32(scene.constants.dt)
    assert k > 5
    meet = k + 2
    w = lib.World(giant_tier_only=True, barrier_timeout_test=True, max_candidates=1)
    w.upload_batch([scene, _meeting_scene(90, meet)])
    # a taped call of three steps runs them kernel by kernel, a longer one replays its graph
    before = k - 1 if steps == "eager" else 1
    w.step(dt, before)
    apart = w.counts()[0]
    with pytest.raises(lib.NansError) as e:
        w.diff_forward(dt, meet - before)
    assert e.value.code == 5 and "timed out" in str(e.value)
    assert w.status() & (1 << 5)
    assert w.counts()[0] > 2 * apart + 2048  # more than any buffer the first steps can have left
    w.close()
