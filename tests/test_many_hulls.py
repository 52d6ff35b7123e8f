"""Steps of so many candidates that the EPAs of hulls of more than eight points run on a thread each (above
60,800 on a GB300), those beyond its polytope handed on to the pair tier: replicas of a few scenes, each
replica's state equal to the oracle's of its scene, bit for bit."""
import numpy as np
import pytest

from helpers import canon
from test_narrow_paths import DT, _hull_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts", [9, 33, 65])
def test_many_hulls(oracle_lib, npts):
    from nans_projekat_gb300 import lib, scenes
    from oracle.portbind import OracleWorld
    seeds = [s for s in range(60) if (scenes.mixed_scene(scenes.SplitMix64(s), 14).hull_npts > 0).any()][:40]
    few = [_hull_scene(scenes, npts, s) for s in seeds]
    reps, steps = 220, 20
    w = lib.World()
    w.upload_batch(few * reps)
    w.batch_step(DT, steps, 10)
    assert w.counts()[0] > 400 * 152 and w.status() == 0
    cubes, spheres, _ = w.download()
    w.close()
    o = OracleWorld(few)
    o.step(DT, steps, 8)
    st = [o.state(i) for i in range(len(few))]
    for got, part in ((cubes, 0), (spheres, 1)):
        for f in ("Position", "Angles", "V", "W"):
            ref = np.concatenate([s[part][f] for s in st]).astype(np.float32)
            g = np.ascontiguousarray(got[f]).reshape(reps, len(ref), 3)
            for r in range(reps):
                assert canon(g[r]) == canon(ref), (f, r)
