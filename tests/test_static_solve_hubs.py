"""nans_solve_contacts_static on lists of more than 1,024 contacts in which bodies have many contacts (on
both sides of the 256 from which a body's contacts are ordered by a bitmap, up to every contact of the
longest list), and with contacts that it skips and reports, against the oracle's sequential solve of the
same list without those, bit for bit."""
import numpy as np
import pytest

from helpers import canon
from test_static_solve_orders import DT, _case

pytestmark = pytest.mark.gpu


def _hubs(rng, n, m, kind):
    ncub, nsph, pos, p = _case(rng, n, m, "random")
    p["Type"], p["IndexA"] = 0, rng.integers(10, ncub, m)
    p["IndexB"] = (p["IndexA"] + 1 - 10) % (ncub - 10) + 10
    if kind == "pair":
        p["IndexA"], p["IndexB"] = 3, 5
    elif kind == "plate":  # body 3 in every contact, on either side
        side = rng.random(m) < 0.5
        p["IndexA"], p["IndexB"] = np.where(side, 3, p["IndexA"]), np.where(side, p["IndexB"], 3)
    else:  # bodies 0, 1, ... of the given numbers of contacts, scattered over the list
        where = rng.permutation(m)
        at = 0
        for body, c in enumerate(kind):
            p["IndexA"][where[at:at + c]] = body
            at += c
    p["PointA"] = pos[p["IndexA"]] + rng.uniform(-0.5, 0.5, (m, 3))
    p["PointB"] = p["PointA"] + rng.uniform(-0.05, 0.05, (m, 3))
    return ncub, nsph, pos, p


@pytest.mark.parametrize("n,m,kind,bad", [
    (40, 1025, (255, 256, 257, 258), 0), (700, 2000, (300, 1, 600, 256, 257), 0), (40, 16384, "pair", 0),
    (9000, 16384, "plate", 0), (9001, 3000, "plate", 0), (95, 16384, "random", 0), (300, 1025, "random", 1),
    (300, 1500, "plate", 1400), (6001, 9000, "random", 37), (40, 1100, "random", 1100)])
def test_solve_equals_the_list_in_order(oracle_lib, n, m, kind, bad):
    import torch
    from nans_projekat_gb300 import lib, scenes
    from oracle.portbind import OracleWorld
    rng = np.random.default_rng(n * 100003 + m)
    ncub, nsph, pos, pairs = _case(rng, n, m, kind) if kind == "random" else _hubs(rng, n, m, kind)
    mass = rng.uniform(0.3, 3.0, n).astype(np.float32)
    moi = (mass * np.float32(0.2)).astype(np.float32)
    vel = rng.normal(0, 1, (n, 3)).astype(np.float32)
    omg = rng.normal(0, 1, (n, 3)).astype(np.float32)
    skip = rng.permutation(m)[:bad]
    kept = np.delete(pairs, skip)
    for i, k in enumerate(skip):
        q = pairs[k:k + 1]
        if i % 4 == 0:
            q["Type"], q["IndexA"], q["IndexB"] = 0, 2, 2  # one body on both sides
        elif i % 4 == 1:
            q["IndexA"] = -1
        elif i % 4 == 2:
            q["Type"], q["IndexA"], q["IndexB"] = 0, 1, ncub
        else:
            q["Type"] = 7
    cubes = scenes._cubes(pos[:ncub], None, mass[:ncub], moi[:ncub], vel[:ncub], omg[:ncub])
    spheres = scenes._spheres(pos[ncub:], 0.5, mass[ncub:], moi[ncub:], vel[ncub:], omg[ncub:])
    sc = scenes.Scene(cubes, spheres, scenes.ground(40.0))
    c, fl = sc.constants, sc.floor[0]
    o = OracleWorld([sc])
    o.hold_contacts(0, [(pos, fl["Position"], kept)])
    o.stage(1, DT)
    o.stage(2, DT)
    oc, os_, _ = o.state(0)
    dev = torch.device("cuda", 0)
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev)
    g_vel, g_omg = t(vel), t(omg)
    args = (t(pos), t(mass), t(moi))
    rec = t(np.frombuffer(pairs.tobytes(), np.uint8).copy())
    floor = np.concatenate([fl["Position"], fl["V"], fl["W"], [fl["Mass"], fl["MOI"]]]).astype(np.float32)
    call = lambda: lib.solve_contacts_static(
        n, ncub, args[0].data_ptr(), args[1].data_ptr(), args[2].data_ptr(), g_vel.data_ptr(), g_omg.data_ptr(), floor,
        rec.data_ptr(), m, c.cr, c.cf, c.iterations, DT, None)
    if bad:
        with pytest.raises(lib.NansError) as e:
            call()
        assert e.value.code == 1 and "skipped" in str(e.value)
    else:
        call()
    for got, f in ((g_vel, "V"), (g_omg, "W")):
        assert canon(got.cpu().numpy()) == canon(np.concatenate([oc[f], os_[f]]).astype(np.float32)), f
