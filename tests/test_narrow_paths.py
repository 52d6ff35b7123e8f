"""The narrowphase's routes against the oracle, bit for bit: a warp per pair for steps of few
candidates, a thread per pair above that with the long runs and the large polytopes on the pair
tier, hulls around the sizes at which a support changes its form; and, on the CPU, the squared
length that stands for the reference's test on a direction's length."""
import numpy as np
import pytest

from helpers import canon

DT = np.float32(1.0 / 60.0)


def test_short_direction_threshold_is_exact():
    """sqrt(x) <= 1e-4f, with a correctly rounded root, exactly for x <= 0x1.5798eep-27."""
    top = np.float32(float.fromhex("0x1.5798eep-27"))
    lim = np.float32(0.0001)
    x = top
    below = []
    for _ in range(1000):
        below.append(x)
        x = np.nextafter(x, np.float32(0))
    x = np.nextafter(top, np.float32(1))
    above = []
    for _ in range(1000):
        above.append(x)
        x = np.nextafter(x, np.float32(1))
    assert (np.sqrt(np.array(below, np.float32)) <= lim).all()
    assert (np.sqrt(np.array(above, np.float32)) > lim).all()


def _hull_scene(scenes, npts, seed):
    """A pile of hulls of npts points, two boxes and a sphere."""
    sc = scenes.mixed_scene(scenes.SplitMix64(seed), 14)
    rng = scenes.SplitMix64(1000 + seed)
    n = np.where(sc.hull_npts > 0, npts, 0).astype(np.int32)
    sc.hull_npts = n
    sc.hull_pts = np.concatenate([scenes.hull_points(rng, npts) for k in n if k]).astype(np.float32)
    return sc


def _compare(batch, steps, step):
    from nans_projekat_gb300 import lib
    from oracle.portbind import OracleWorld
    w = lib.World()
    w.upload_batch(batch)
    step(w, steps)
    got = w.get_state_arrays()
    pairs = [w.pairs(i) for i in (0, len(batch) - 1)]
    assert w.status() == 0
    w.close()
    o = OracleWorld(batch)
    o.step(DT, steps, 8)
    st = [o.state(i) for i in range(len(batch))]
    for a, f in zip(got, ("Position", "Angles", "V", "W")):
        ref = np.concatenate([c[f] for c, _, _ in st] + [s[f] for _, s, _ in st]).astype(np.float32)
        assert canon(a) == canon(ref), f
    for p, i in zip(pairs, (0, len(batch) - 1)):
        op = o.pairs(i)
        for f in ("Type", "IndexA", "IndexB", "PointA", "PointB", "N"):
            assert canon(p[f]) == canon(op[f]), f


@pytest.mark.gpu
@pytest.mark.parametrize("n_scenes,lo,hi", [(1, 4, 4), (1, 130, 130), (1, 256, 256), (1, 300, 300), (40, 30, 60),
                                             (60, 40, 80)])
def test_few_and_many_pairs(oracle_lib, n_scenes, lo, hi):
    """One scene of 4 bodies (10 pairs) up to candidates on both sides of the count (2,432 on a
    GB300) at which a step leaves the warp-per-pair form, past the impact of the projectile; contact
    lists on both sides of the lengths (128 and 256) at which the solver labels its waves otherwise."""
    from nans_projekat_gb300 import scenes
    batch = scenes.stack_batch(n_scenes, seed=31, lo=lo, hi=hi)
    _compare(batch, 45, lambda w, n: w.step(DT, n))


@pytest.mark.gpu
@pytest.mark.parametrize("npts", [4, 7, 8, 9, 31, 32, 33, 65])
@pytest.mark.parametrize("n_scenes", [1, 70])
def test_hull_sizes(oracle_lib, npts, n_scenes):
    """Hulls of fewer and more points than a thread's registers (8) and a warp's lanes (32) hold,
    on the warp-per-pair form (one scene) and the thread-per-pair one (70)."""
    from nans_projekat_gb300 import scenes
    batch = [_hull_scene(scenes, npts, 5 + i) for i in range(n_scenes)]
    _compare(batch, 30, lambda w, n: w.batch_step(DT, n, 10))


@pytest.mark.gpu
@pytest.mark.parametrize("n_scenes,bodies", [(1, 92), (30, 75)])
def test_full_blocks_of_the_cull(n_scenes, bodies):
    """With every pair kept, a block of the cull's placement lists its candidates in more than one
    round (8,192 pairs a block against a list of 4,096): the same contacts and states as the culled
    run, for one block's pairs and for several blocks'."""
    from nans_projekat_gb300 import lib, scenes
    batch = scenes.stack_batch(n_scenes, seed=17, lo=bodies, hi=bodies)
    out = []
    for every in (False, True):
        w = lib.World(all_pairs=every, max_candidates=2 * n_scenes * bodies * bodies)
        w.upload_batch(batch)
        w.batch_step(DT, 12, 6)
        pairs = [w.pairs(i) for i in range(n_scenes)]
        out.append((w.get_state_arrays(), pairs, w.counts(), w.status()))
        w.close()
    assert out[1][2][0] > 4096 * (1 if n_scenes == 1 else 10) and out[0][2][1] == out[1][2][1]
    assert out[0][3] == 0 and out[1][3] == 0
    for a, b in zip(out[0][0], out[1][0]):
        assert canon(a) == canon(b)
    for p, q in zip(out[0][1], out[1][1]):
        for f in ("Type", "IndexA", "IndexB", "PointA", "PointB", "N"):
            assert canon(p[f]) == canon(q[f])
