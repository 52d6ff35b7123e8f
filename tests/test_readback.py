"""Reading a world back on both sides of the size up to which the kernels write straight to
page-locked memory (64 KB): records, state arrays and contact lists against the oracle bit for bit,
with the last step's velocities applied once, whatever is read first and however often."""
import ctypes

import numpy as np
import pytest

from helpers import canon

pytestmark = pytest.mark.gpu
DT = np.float32(1.0 / 60.0)


def _scene(scenes, n, spheres):
    return scenes.random_scene(seed=n, n_boxes=n - spheres, n_spheres=spheres, extent=12.0)


# 244 bytes a cube and floor, 148 a sphere; 12 bytes a body and array
@pytest.mark.parametrize("n,spheres", [(2, 1), (33, 3), (267, 0), (268, 0), (500, 260), (1365, 300), (1366, 300)])
def test_every_way_of_reading_gives_the_oracles_state(oracle_lib, n, spheres):
    from nans_projekat_gb300 import lib, scenes
    from oracle.portbind import OracleWorld
    sc = _scene(scenes, n, spheres)
    o = OracleWorld([sc])
    worlds = [lib.World() for _ in range(3)]
    for w in worlds:
        w.upload(sc)
    for k in range(2):
        o.step(DT, 1)
        for w in worlds:
            w.step(DT, 1)
        oc, os_, _ = o.state(0)
        want = [canon(np.concatenate([oc[f], os_[f]]).astype(np.float32)) for f in ("Position", "Angles", "V", "W")]
        # records first, arrays first (twice), and arrays in parts: the velocities before the positions
        c, s, _ = worlds[0].download()
        assert [canon(np.concatenate([c[f], s[f]]).astype(np.float32)) for f in ("Position", "Angles", "V", "W")] == want
        for _ in range(2):
            assert [canon(a) for a in worlds[1].get_state_arrays()] == want
        parts = [np.zeros((n, 3), np.float32) for _ in range(4)]
        for q in (2, 3, 0, 1):
            worlds[2].lib.nans_world_get_state_arrays(
                worlds[2].h, *[a.ctypes.data if i == q else None for i, a in enumerate(parts)])
        assert [canon(a) for a in parts] == want
        again = worlds[1].download()
        assert canon(again[0]) == canon(c) and canon(again[1]) == canon(s)
    for w in worlds:
        w.close()


@pytest.mark.parametrize("cap", [0, 1, 255, 256, 257, 682, 683, 2000])
def test_contact_lists_up_to_any_length(oracle_lib, cap):
    """682 records fit the page-locked buffer."""
    from nans_projekat_gb300 import lib, scenes
    from nans_projekat_gb300.types import PAIR_DTYPE
    from oracle.portbind import OracleWorld
    sc = scenes.stack_scene_random(scenes.SplitMix64(5), 1000)
    o = OracleWorld([sc])
    o.step(DT, 10)
    want = o.pairs(0)
    assert len(want) > 683
    w = lib.World()
    w.upload(sc)
    w.step(DT, 10)
    out = np.zeros(max(1, cap), PAIR_DTYPE)
    n = ctypes.c_uint32()
    assert w.lib.nans_get_pairs(w.h, 0, ctypes.c_void_p(out.ctypes.data), cap, ctypes.byref(n)) == 0
    assert n.value == len(want)
    m = min(cap, len(want))
    for f in ("Type", "IndexA", "IndexB", "PointA", "PointB", "N"):
        assert canon(np.ascontiguousarray(out[:m][f])) == canon(np.ascontiguousarray(want[:m][f])), f
    w.close()
