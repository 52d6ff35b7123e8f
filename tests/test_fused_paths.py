"""Worlds that take the fused per-scene step (up to 14 bodies a scene, up to two scenes per SM: 304 on a
GB300), each checked to do so, against the oracle bit for bit: scenes of all
sizes, one and many a launch, with hulls, with every pair kept, with EPAs beyond the warp tier among them;
and the line on whose other side a world takes the staged kernels."""
import numpy as np
import pytest

from helpers import canon

pytestmark = pytest.mark.gpu
DT = np.float32(1.0 / 60.0)
FUSED = (5, 5)  # sweep, scene step, block EPA, giant EPA, late solve


def _hulls(npts, n_scenes):
    """Scenes of 4 to 14 bodies of which some are hulls of npts points."""
    from nans_projekat_gb300 import scenes
    rng, out, seed = scenes.SplitMix64(npts), [], 0
    while len(out) < n_scenes:
        seed += 1
        sc = scenes.mixed_scene(scenes.SplitMix64(1000 * npts + seed), 4 + seed % 11)
        if not (sc.hull_npts > 0).any():
            continue
        sc.hull_npts = np.where(sc.hull_npts > 0, npts, 0).astype(np.int32)
        sc.hull_pts = np.concatenate([scenes.hull_points(rng, npts) for k in sc.hull_npts if k]).astype(np.float32)
        out.append(sc)
    return out


def _batch(kind):
    from nans_projekat_gb300 import scenes
    if kind == "uneven":
        return scenes.stack_batch(100, seed=40, lo=2, hi=14), {}
    if kind == "most":
        return scenes.stack_batch(304, seed=41, lo=14, hi=14), {}
    if kind == "one":
        return scenes.stack_batch(1, seed=42, lo=14, hi=14), {}
    if kind == "mixed":
        return scenes.mixed_batch(60, seed=43, lo=4, hi=14), {}
    if kind == "all_pairs":
        return scenes.stack_batch(80, seed=44, lo=3, hi=14), dict(all_pairs=True)
    return _hulls(int(kind), 40), {}


@pytest.mark.parametrize("kind", ["uneven", "most", "one", "mixed", "all_pairs", "7", "31", "33", "65"])
def test_fused_batches_match_oracle(oracle_lib, kind):
    from nans_projekat_gb300 import lib
    from oracle.portbind import OracleWorld
    batch, flags = _batch(kind)
    o = OracleWorld(batch)
    worlds = [lib.World(fused_step=True, **flags) for _ in range(2)]
    for w in worlds:
        w.upload_batch(batch)
        assert w.launches_per_step() == FUSED
    for _ in range(3):
        o.step(DT, 15, 8)
        worlds[0].step(DT, 15)
        worlds[1].batch_step(DT, 15, 5)
        for w in worlds:
            cubes, spheres, _ = state = w.download()
            for i in range(len(batch)):
                oc, os_, _ = o.state(i)
                c, s, _ = w.scene_state(i, state)
                for f in ("Position", "Angles", "V", "W"):
                    assert canon(c[f]) == canon(oc[f]) and canon(s[f]) == canon(os_[f]), (i, f)
                p, q = w.pairs(i), o.pairs(i)
                for f in ("Type", "IndexA", "IndexB", "PointA", "PointB", "N"):
                    assert canon(p[f]) == canon(q[f]), (i, f)
            assert w.status() == 0
    staged = lib.World(**flags, max_candidates=60000)
    staged.upload_batch(batch)
    staged.batch_step(DT, 45, 5)
    assert staged.launches_per_step() != FUSED and staged.counts() == worlds[0].counts() == worlds[1].counts()
    for w in worlds + [staged]:
        w.close()


# stacks whose EPAs outgrow the warp tier once within 40 steps (504, 506 and 894 faces): seed, bodies
LATE = ((134709, 7), (50543, 13), (185767, 14))


@pytest.mark.parametrize("giant", [False, True])
@pytest.mark.parametrize("graph", [1, 5])
def test_late_scenes_among_others(oracle_lib, graph, giant):
    """Scenes with an EPA beyond the warp tier, which the fused launch leaves to the large tiers and the late
    solve (behind a condition in its graphs), two of each between scenes that have none."""
    from nans_projekat_gb300 import lib, scenes
    from oracle.portbind import OracleWorld
    late = [scenes.stack_scene_random(scenes.SplitMix64(s), n) for s, n in LATE]
    batch = scenes.stack_batch(30, seed=45, lo=2, hi=14)
    at = [4 * k + 1 for k in range(6)]
    for i, sc in zip(at, late * 2):
        batch.insert(i, sc)
    w = lib.World(fused_step=True, giant_tier_only=giant)
    w.upload_batch(batch)
    assert w.launches_per_step() == FUSED
    o = OracleWorld(batch)
    for _ in range(4):
        w.batch_step(DT, 10, graph)
        o.step(DT, 10, 8)
        state = w.download()
        for i in range(len(batch)):
            oc, os_, _ = o.state(i)
            c, s, _ = w.scene_state(i, state)
            for f in ("Position", "Angles", "V", "W"):
                assert canon(c[f]) == canon(oc[f]) and canon(s[f]) == canon(os_[f]), (i, f)
    e = w.epa_stats()
    assert e["slow_epas"] == 6 and (e["giant_tier"] == 6) == giant and w.status() == 0
    w.close()


@pytest.mark.parametrize("n_scenes,bodies,fused", [(1, 14, True), (1, 15, False), (304, 5, True), (305, 5, False)])
def test_the_line(n_scenes, bodies, fused):
    from nans_projekat_gb300 import lib, scenes
    w = lib.World(fused_step=True)
    w.upload_batch(scenes.stack_batch(n_scenes, seed=46, lo=bodies, hi=bodies))
    assert (w.launches_per_step() == FUSED) == fused
    w.step(DT, 3)
    assert w.status() == 0
    w.close()
