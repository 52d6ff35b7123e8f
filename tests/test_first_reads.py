"""A world's first reads, which go through pageable memory, give what its later ones through page-locked
memory give: every call that reads something back, as the first, second, third and fourth of its world."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DT = np.float32(1.0 / 60.0)


def _calls(w):
    buf = tuple(np.full((w.n_bodies, 3), 7.0, np.float32) for _ in range(4))
    return dict(arrays=lambda: w.get_state_arrays(out=buf), records=w.download, pairs=lambda: (w.pairs(0), w.pairs(1)),
                counts=w.counts, step=lambda: w.step(DT, 1), batch=lambda: w.batch_step(DT, 1, 1),
                diff=lambda: w.diff_forward(DT, 2))


@pytest.mark.parametrize("first", ["arrays", "records", "pairs", "step", "batch", "diff"])
def test_first_reads(first):
    from nans_projekat_gb300 import lib, scenes
    batch = scenes.stack_batch(2, seed=12, lo=20, hi=30)
    # where the boxes rest and touch
    w = lib.World()
    w.upload_batch(batch)
    w.step(DT, 12)
    start = w.get_state_arrays()
    w.close()
    seen = []
    for before in (0, 1, 2, 3, 20):
        w = lib.World()
        w.upload_batch(batch)
        w.set_state_arrays(*start)
        for _ in range(before):
            w.pairs(0)  # a read that changes nothing
        _calls(w)[first]()
        # the steps a call does not take itself, so that every call ends in the same state
        w.step(DT, 3 - dict(step=1, batch=1, diff=2).get(first, 0))
        c = _calls(w)
        p, q = c["pairs"]()
        assert len(p) > 0 and len(q) > 0
        cubes, spheres, floors = c["records"]()
        seen.append([x.tobytes() for x in (p, q, cubes, spheres, floors) + tuple(c["arrays"]())] + [w.counts()])
        w.close()
    for s in seen[1:]:
        assert s == seen[0]
