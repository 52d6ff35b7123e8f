"""nans_solve_contacts_static on contact lists of any order against the oracle's sequential solve
of the same list, bit for bit: sizes around the block's threads, around the length from which a list
is ordered by a launch of its own, and around the number of bodies whose velocities fit shared
memory, one body in every contact, repeated contacts of one pair, and the entry point's limits."""
import numpy as np
import pytest

from helpers import canon

pytestmark = pytest.mark.gpu
DT = np.float32(1.0 / 60.0)


def _case(rng, n, m, kind):
    from nans_projekat_gb300.types import PAIR_DTYPE
    ncub = max(2, (3 * n) // 4)
    nsph = n - ncub
    pos = rng.uniform(-4, 4, (n, 3)).astype(np.float32)
    a = rng.integers(0, n, m)
    b = rng.integers(0, n + max(1, n // 8), m)  # beyond n: the ground
    if kind == "star":
        a[:] = 1
    elif kind == "repeated":
        a[:], b[:] = np.sort(rng.integers(0, 2, m)), 1
        a[:] = 0
    elif kind == "chain":
        a[:] = np.arange(m) % (n - 1)
        b[:] = a + 1
    floor = (b >= n) | (a == b)
    sa, sb = a >= ncub, (b >= ncub) & ~floor
    swap = sa & ~sb & ~floor  # a cube-sphere contact names the cube first
    a, b = np.where(swap, b, a), np.where(swap, a, b)
    sa, sb = np.where(swap, False, sa), np.where(swap, True, sb)
    p = np.zeros(m, PAIR_DTYPE)
    p["Type"] = np.where(floor, np.where(sa, 4, 2), np.where(sa, 3, np.where(sb, 1, 0)))
    p["IndexA"] = np.where(sa, a - ncub, a)
    p["IndexB"] = np.where(floor, p["IndexA"], np.where(sb, b - ncub, b))
    nrm = rng.standard_normal((m, 3))
    p["N"] = nrm / np.linalg.norm(nrm, axis=1, keepdims=True)
    p["PointA"] = pos[a] + rng.uniform(-0.5, 0.5, (m, 3))
    p["PointB"] = p["PointA"] + rng.uniform(-0.05, 0.05, (m, 3))
    if m > 3:
        p["N"][m // 2] = 0.0  # the solve takes the direction between the bodies instead
    return ncub, nsph, pos, p


@pytest.mark.parametrize("n,m,kind", [(2, 1, "random"), (3, 7, "random"), (40, 511, "random"), (300, 512, "random"),
                                      (300, 513, "random"), (60, 2000, "star"), (5, 400, "repeated"),
                                      (1500, 1499, "chain"), (6000, 9000, "random"), (6001, 9000, "random"),
                                      (6001, 500, "random"), (300, 1024, "random"), (300, 1025, "random"),
                                      (9000, 2500, "random"), (9001, 2500, "random"), (700, 1025, "chain"),
                                      (4913, 16384, "random"), (16384, 16384, "random")])
def test_solve_equals_the_list_in_order(oracle_lib, n, m, kind):
    import torch
    from nans_projekat_gb300 import lib, scenes
    from oracle.portbind import OracleWorld
    rng = np.random.default_rng(n * 100003 + m)
    ncub, nsph, pos, pairs = _case(rng, n, m, kind)
    mass = rng.uniform(0.3, 3.0, n).astype(np.float32)
    moi = (mass * np.float32(0.2)).astype(np.float32)
    vel = rng.normal(0, 1, (n, 3)).astype(np.float32)
    omg = rng.normal(0, 1, (n, 3)).astype(np.float32)
    cubes = scenes._cubes(pos[:ncub], None, mass[:ncub], moi[:ncub], vel[:ncub], omg[:ncub])
    spheres = scenes._spheres(pos[ncub:], 0.5, mass[ncub:], moi[ncub:], vel[ncub:], omg[ncub:]) if nsph else \
        scenes._spheres(np.zeros((0, 3)), 0.5, np.zeros(0), np.zeros(0))
    sc = scenes.Scene(cubes, spheres, scenes.ground(40.0))
    c = sc.constants
    o = OracleWorld([sc])
    fl = sc.floor[0]
    o.hold_contacts(0, [(pos, fl["Position"], pairs)])
    o.stage(1, DT)
    o.stage(2, DT)
    oc, os_, _ = o.state(0)
    dev = torch.device("cuda", 0)
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev)
    g_vel, g_omg = t(vel), t(omg)
    args = (t(pos), t(mass), t(moi))
    rec = t(np.frombuffer(pairs.tobytes(), np.uint8).copy())
    floor = np.concatenate([fl["Position"], fl["V"], fl["W"], [fl["Mass"], fl["MOI"]]]).astype(np.float32)
    lib.solve_contacts_static(n, ncub, args[0].data_ptr(), args[1].data_ptr(), args[2].data_ptr(), g_vel.data_ptr(),
                              g_omg.data_ptr(), floor, rec.data_ptr(), m, c.cr, c.cf, c.iterations, DT, None)
    for got, f in ((g_vel, "V"), (g_omg, "W")):
        assert canon(got.cpu().numpy()) == canon(np.concatenate([oc[f], os_[f]]).astype(np.float32)), f
