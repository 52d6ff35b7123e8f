"""The same rollout gives the same gradients, bit for bit: scenes whose solve takes one warp, two (from 128
bodies), eight (above 512), and the late pass's four, lists of one and of several chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DT = np.float32(1.0 / 60.0)


@pytest.mark.parametrize("scenes_bodies,steps", [((20, 33), 25), ((40, 200), 3), ((40, 200), 20), ((1, 600), 10)])
def test_gradients_repeat(scenes_bodies, steps):
    from nans_projekat_gb300 import lib, scenes
    n, bodies = scenes_bodies
    batch = scenes.stack_batch(n, seed=23, lo=bodies, hi=bodies)
    w = lib.World()
    w.upload_batch(batch)
    w.batch_step(DT, 3, 1)
    start = w.get_state_arrays()
    loss = np.random.default_rng(2).standard_normal((4, w.n_bodies, 3)).astype(np.float32)
    first = None
    for _ in range(6):
        w.set_state_arrays(*start)
        w.diff_forward(DT, steps)
        g = w.diff_backward(*loss)
        assert np.abs(g["restitution"]).max() > 0 and np.abs(g["friction"]).max() > 0
        if first is None:
            first = {k: v.copy() for k, v in g.items()}
        for k in first:
            assert g[k].tobytes() == first[k].tobytes(), k
    w.close()
