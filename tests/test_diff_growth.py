"""The taped step's graph and its growth: bodies that meet after some steps need more candidate slots
than the first step allocated, so a step replayed from the graph is put back, run again with larger
buffers and taped; the rollout equals one whose buffers held every pair from the start."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DT = np.float32(1.0 / 60.0)


def _meeting_scene(n):
    """n heavy unit boxes on a sphere of 240 m that move 12 m a step to its centre: apart until step 20,
    on top of each other at step 21."""
    from nans_projekat_gb300 import scenes
    rng = np.random.default_rng(5)
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    pos = 240.0 * d + np.array([0.0, 400.0, 0.0])
    mass = rng.uniform(500.0, 2000.0, n)
    cubes = scenes._cubes(pos, None, mass, mass / 6.0, vel=-12.0 * d / float(DT))
    spheres = scenes._spheres([[30.0, 5.0, 0.0]], 0.5, 1.0, 0.1)
    return scenes.Scene(cubes, spheres, scenes.ground(60.0))


@pytest.mark.parametrize("steps", [3, 21])
def test_growth_inside_a_taped_rollout(steps):
    from nans_projekat_gb300 import lib
    sc = _meeting_scene(70)
    g = np.random.default_rng(1).standard_normal((4, 71, 3)).astype(np.float32)
    out = []
    for cap in (0, 1):
        w = lib.World(max_candidates=cap)
        w.upload(sc)
        w.diff_forward(DT, steps)
        counts = w.counts()
        grads = w.diff_backward(*g)
        assert w.diff_tape_info()[0] == steps
        out.append((w.get_state_arrays(), grads, counts))
        w.close()
    if steps > 20:
        assert out[0][2][0] > 1400  # more than the 1,024 and a quarter the first step left room for
    assert out[0][2] == out[1][2]
    for a, b in zip(out[0][0], out[1][0]):
        assert a.tobytes() == b.tobytes()
    for k in out[0][1]:
        a, b = out[0][1][k], out[1][1][k]
        assert np.allclose(a, b, rtol=1e-5, atol=1e-5 * max(1e-30, float(np.abs(a).max()))), k
