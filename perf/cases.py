"""The work that users of the physics step have it do, as cases that can be timed and compared.

A case is a dict of plain values; its "kind" names the way the library is called:

* frame   one scene through the drop-in path, once per rendered frame: the host hands its body
          records over, one step runs, the records and the frame's contact list come back.
* single  one scene stepped many times between two looks at its state (a replay, a preview), with
          the staged kernels or with the fused per-scene step.
* batch   many independent scenes of uneven sizes (a learner's environments, a parameter sweep):
          the state goes in as arrays, the batched path replays its graph, the state comes back.
          With boxes only, or with boxes, spheres and convex hulls; with or without warm starting.
* diff    the differentiable rollout: a taped forward and the gradients of a loss of its final
          state, as one iteration of an optimiser calls it.
* solve   the allocation-free contact solve on device buffers that the caller owns.

Everything is single precision; the step is defined bit for bit, so it has no other type. The
stepping cases start a few steps (or a second of simulated time) after the scenes were made, when
the stacks rest on each other or have begun to fall.
"""
import math

import numpy as np
import torch

from nans_projekat_gb300 import lib, scenes
from nans_projekat_gb300.types import CC, CF, CS, PAIR_DTYPE, SF, SS

DT = np.float32(1.0 / 60.0)
STACKS = dict(lo=4, hi=256)   # body counts of the batched stacks, log-uniform
MIXED = dict(lo=8, hi=128)    # body counts of the scenes with hulls, uniform


def listed():
    return [
        # The reference's own use: one small scene, one step per rendered frame, records in and out.
        dict(name="frame_stack9", kind="frame", scene="stack9", bodies=9, constants="config", settle=20),
        # The same kind of host with an ordinary pile and the reference's solver literals.
        dict(name="frame_stack60", kind="frame", scene="stack", bodies=60, constants="reference", settle=30),
        # A second of a small scene in one call, with the fused step that is meant for it.
        dict(name="single_stack9_fused", kind="single", scene="stack9", bodies=9, spheres=1, steps=60, settle=0,
             fused=True),
        # One large scene (4,096 boxes, 512 spheres): the plain path where the pair space is largest.
        dict(name="single_random4608", kind="single", scene="random", bodies=4608, spheres=512, steps=4, settle=2,
             fused=False),
        # A learner's environments, one step per call: the state crosses the host link every step.
        dict(name="batch_1000_by_step", kind="batch", scene="stack", scenes=1000, steps=1, settle=5, warm=False,
             **STACKS),
        # The headline workload: 16,384 uneven stacks, twenty steps per call.
        dict(name="batch_16384", kind="batch", scene="stack", scenes=16384, steps=20, settle=5, warm=False,
             **STACKS),
        # Convex hulls, spheres and boxes together.
        dict(name="batch_hulls_777", kind="batch", scene="mixed", scenes=777, steps=10, settle=10, warm=False,
             **MIXED),
        # Warm starting, a second into the run, when the stacks have come apart.
        dict(name="batch_warm_2048", kind="batch", scene="stack", scenes=2048, steps=10, settle=60, warm=True,
             **STACKS),
        # The differentiated configuration: 1,024 scenes of 33 bodies, 120 steps, forward and backward.
        dict(name="diff_1024x33", kind="diff", scene="grid", scenes=1024, lo=33, hi=33, steps=120),
        # Gradients through uneven scenes with hulls, a short horizon (one checkpointed segment).
        dict(name="diff_hulls_301", kind="diff", scene="mixed", scenes=301, steps=20, **MIXED),
        # The caller-owned solve: an ordinary pile, and one near the entry point's limit.
        dict(name="solve_pile_125", kind="solve", nx=5, ny=5, nz=5, spheres=25, iterations=10),
        dict(name="solve_pile_4913", kind="solve", nx=17, ny=17, nz=17, spheres=601, iterations=10),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("frame", "single", "single", "batch", "batch", "batch", "diff", "solve"))
    if kind == "frame":
        return dict(kind=kind, scene="stack", bodies=_log_int(rng, 3, 256),
                    constants=rng.choice(("config", "reference")), settle=rng.randint(3, 60))
    if kind == "single":
        if rng.random() < 0.5:
            return dict(kind=kind, scene="stack", bodies=_log_int(rng, 3, 256), spheres=1,
                        steps=_log_int(rng, 4, 120), settle=rng.randint(0, 30), fused=rng.random() < 0.5)
        n = _log_int(rng, 200, 4608)
        return dict(kind=kind, scene="random", bodies=n, spheres=rng.randint(0, n // 8), steps=rng.randint(1, 4),
                    settle=rng.randint(0, 8), fused=False)
    if kind == "batch":
        scene = rng.choice(("stack", "stack", "mixed"))
        n = _log_int(rng, 32, 8192 if scene == "stack" else 1024)
        lo = rng.randint(4, 12)
        return dict(kind=kind, scene=scene, scenes=n, lo=lo, hi=_log_int(rng, 24, 256 if scene == "stack" else 128),
                    steps=_log_int(rng, 1, 20), settle=rng.randint(3, 60), warm=rng.random() < 0.25)
    if kind == "diff":
        scene = rng.choice(("grid", "mixed", "stack"))
        n = _log_int(rng, 16, 1024 if scene == "grid" else 256)
        lo, hi = (33, 33) if scene == "grid" else (rng.randint(4, 12), _log_int(rng, 24, 128))
        return dict(kind=kind, scene=scene, scenes=n, lo=lo, hi=hi, steps=_log_int(rng, 4, 60))
    nx, ny, nz = (rng.randint(2, 17) for _ in range(3))
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, spheres=rng.randint(0, nx * ny * nz // 4),
                iterations=rng.choice((10, 10, 70)))


# ---- scenes ------------------------------------------------------------------------------


def _constants(case):
    return scenes.Constants.reference_defaults() if case.get("constants") == "reference" else scenes.Constants()


def _one_scene(case, seed):
    if case["scene"] == "stack9":
        return scenes.stack_scene(seed, _constants(case))
    if case["scene"] == "stack":
        return scenes.stack_scene_random(scenes.SplitMix64(seed), case["bodies"], _constants(case))
    # the density of the 4,608-body scene in its 64 m box, whatever the body count
    extent = 64.0 * (case["bodies"] / 4608.0) ** (1.0 / 3.0)
    return scenes.random_scene(seed, case["bodies"] - case["spheres"], case["spheres"], extent)


def _many_scenes(case, seed):
    if case["scene"] == "grid":
        return scenes.grid_stack_batch(case["scenes"], seed)
    # the sizes of a case's scenes are its own, what is in them the seed's
    n, lo, hi = case["scenes"], case["lo"], case["hi"]
    sizes = scenes.SplitMix64(n)
    rng = scenes.SplitMix64(seed)
    if case["scene"] == "stack":
        counts = np.floor(np.exp(sizes.uniform(n, math.log(lo), math.log(hi + 1))))
        return [scenes.stack_scene_random(rng, int(k)) for k in np.clip(counts, lo, hi)]
    return [scenes.mixed_scene(rng, int(k)) for k in np.floor(sizes.uniform(n, lo, hi + 1))]


def _pinned(n):
    return tuple(torch.empty((n, 3), dtype=torch.float32, pin_memory=True).numpy() for _ in range(4))


# ---- the contact solve's inputs: a jittered grid of bodies, touching their neighbours -----


def _pile(case, seed):
    """Bodies (the cubes, then the spheres), the contacts between grid neighbours and with the
    ground in the reference's order (CC, CF, SF, CS, SS), and the ground, as numpy arrays."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    nsph = case["spheres"]
    ncub = n - nsph
    cell = np.stack(np.meshgrid(np.arange(ny), np.arange(nx), np.arange(nz), indexing="ij"), -1).reshape(n, 3)[:, [1, 0, 2]]
    body = rng.permutation(n)  # the body in each cell: the spheres lie anywhere in the pile
    pos = np.empty((n, 3), np.float32)
    pos[body] = cell + np.array([0.0, 0.49, 0.0]) + rng.uniform(-0.02, 0.02, (n, 3))
    vel = rng.normal(0.0, 0.5, (n, 3)).astype(np.float32)
    omg = rng.normal(0.0, 0.5, (n, 3)).astype(np.float32)
    mass = rng.uniform(0.25, 3.0, n).astype(np.float32)
    moi = (mass * np.float32(1.0 / 6.0)).astype(np.float32)
    at = np.full((ny, nx, nz), -1)
    at[cell[:, 1], cell[:, 0], cell[:, 2]] = body
    near = [np.stack([at[:, :-1].ravel(), at[:, 1:].ravel()], 1), np.stack([at[:-1].ravel(), at[1:].ravel()], 1),
            np.stack([at[:, :, :-1].ravel(), at[:, :, 1:].ravel()], 1)]
    pr = np.concatenate(near)
    pr = np.sort(pr, axis=1)  # a cube's index is below a sphere's, the lower index first
    ground = np.sort(at[0].ravel())
    sph_a, sph_b = pr[:, 0] >= ncub, pr[:, 1] >= ncub
    rows = []
    for kind, sel in ((CC, ~sph_b), (CF, None), (SF, None), (CS, ~sph_a & sph_b), (SS, sph_a)):
        if kind in (CF, SF):
            g = ground[(ground >= ncub) == (kind == SF)]
            ab = np.stack([g, np.full_like(g, -1)], 1)
        else:
            ab = pr[sel]
            ab = ab[np.lexsort((ab[:, 1], ab[:, 0]))]
        rows.append(np.concatenate([np.full((len(ab), 1), kind), ab], 1))
    rows = np.concatenate(rows)
    m = len(rows)
    a, b = rows[:, 1], rows[:, 2]
    floor_c = b < 0
    pb = np.where(floor_c[:, None], pos[a] * np.array([1, 0, 1], np.float32), pos[np.maximum(b, 0)])
    d = pos[a].astype(np.float64) - pb
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    mid = np.where(floor_c[:, None], pb, 0.5 * (pos[a].astype(np.float64) + pb)) + rng.uniform(-0.3, 0.3, (m, 3)) * (1 - np.abs(d))
    depth = rng.uniform(0.0, 0.03, (m, 1))
    pairs = np.zeros(m, PAIR_DTYPE)
    pairs["Type"] = rows[:, 0]
    pairs["N"] = -d
    pairs["PointA"] = mid - 0.5 * depth * d
    pairs["PointB"] = mid + 0.5 * depth * d
    pairs["IndexA"] = np.where(a >= ncub, a - ncub, a)
    pairs["IndexB"] = np.where(floor_c, pairs["IndexA"], np.where(b >= ncub, b - ncub, b))
    ground_rec = np.array([0.0, -0.5, 0.0, 0, 0, 0, 0, 0, 0, 1e5, 1e5 / 12.0 * 800.0], np.float32)
    return pos, vel, omg, mass, moi, pairs, ground_rec, ncub


# ---- prepare and run ---------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        pos, vel, omg, mass, moi, pairs, ground, ncub = _pile(case, seed)
        dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
        st = dict(kind=kind, n=len(pos), ncub=ncub, pos=dev(pos), vel0=dev(vel), omg0=dev(omg), mass=dev(mass),
                  moi=dev(moi), pairs=dev(np.frombuffer(pairs.tobytes(), np.uint8).copy()), npairs=len(pairs),
                  ground=ground, iterations=case["iterations"])
        st["vel"], st["omg"] = torch.empty_like(st["vel0"]), torch.empty_like(st["omg0"])
        torch.cuda.synchronize()
        return st
    if kind in ("frame", "single"):
        w = lib.World(fused_step=bool(case.get("fused")))
        w.upload(_one_scene(case, seed))
        if case["settle"]:
            w.step(DT, case["settle"])
        if kind == "frame":
            w.step(DT, 1)
            cubes, spheres, _ = w.download()
            # the host's own list of the frame's contacts, for its debug drawing
            return dict(kind=kind, world=w, cubes=cubes, spheres=spheres,
                        contacts=np.zeros(64 + 8 * case["bodies"], PAIR_DTYPE))
    else:
        w = lib.World(warm_start=bool(case.get("warm")))
        w.upload_batch(_many_scenes(case, seed))
        if case.get("settle"):
            w.batch_step(DT, case["settle"], 1)
    st = dict(kind=kind, world=w, steps=case["steps"], start=_pinned(w.n_bodies), out=_pinned(w.n_bodies))
    w.get_state_arrays(out=st["start"])
    if kind == "batch":
        w.set_state_arrays(*st["start"])
        w.prepare(DT, st["steps"])
    if kind == "diff":
        rng = np.random.default_rng(seed)
        st["grads"] = [rng.standard_normal((w.n_bodies, 3)).astype(np.float32) for _ in range(4)]
    return st


def _records(rec):
    return rec.view(np.float32).reshape(len(rec), -1)


def run(state):
    kind = state["kind"]
    if kind == "solve":
        vel, omg = state["vel"], state["omg"]
        vel.copy_(state["vel0"])
        omg.copy_(state["omg0"])
        lib.solve_contacts_static(state["n"], state["ncub"], state["pos"].data_ptr(), state["mass"].data_ptr(),
                                  state["moi"].data_ptr(), vel.data_ptr(), omg.data_ptr(), state["ground"],
                                  state["pairs"].data_ptr(), state["npairs"], 0.2, 0.5, state["iterations"], DT,
                                  torch.cuda.current_stream().cuda_stream)
        return dict(velocity=vel, omega=omg)
    w = state["world"]
    if kind == "frame":
        w.set_state(state["cubes"], state["spheres"], keep_model=True)
        w.step(DT, 1)
        cubes, spheres, _ = w.download()
        p = w.pairs(0)
        state["contacts"][:len(p)] = p
        state["contacts"][len(p):] = 0
        p = state["contacts"]
        out = dict(cubes=_records(cubes), spheres=_records(spheres))
        out.update((f, p[f]) for f in ("Type", "IndexA", "IndexB", "PointA", "PointB", "N"))
        return out
    w.set_state_arrays(*state["start"])
    out = dict(zip(("position", "angles", "velocity", "omega"), state["out"]))
    if kind == "single":
        w.step(DT, state["steps"])
        w.get_state_arrays(out=state["out"])
    elif kind == "batch":
        w.batch_step(DT, state["steps"], state["steps"])
        w.get_state_arrays(out=state["out"])
    else:
        w.diff_forward(DT, state["steps"])
        # the gradients first: the tape belongs to the state that the forward left
        out.update(w.diff_backward(*state["grads"]))
        w.get_state_arrays(out=state["out"])
    return out


# ---- what a pass cannot do without ---------------------------------------------------------


def _bodies(case):
    if "scenes" not in case:
        return float(case["bodies"])
    lo, hi = case["lo"], case["hi"]
    if lo == hi:
        return float(case["scenes"]) * lo
    mean = (lo + hi) / 2.0 if case["scene"] == "mixed" else (hi - lo) / math.log(hi / lo)
    return case["scenes"] * mean


def work(case):
    """Bytes: each body's state in and out with its mass, inertia and scale, the records and
    contacts of a frame, the gradients of a rollout. Operations, in single precision: per body and
    step about 500 (RK4, the model matrix, eight vertices, the box); per contact about 2,500 (a GJK
    of six and an EPA of three rounds of two eight-vertex supports, ten solver iterations); a
    contact per body, as the stacks have. The adjoint's share is 300 a contact and step."""
    if case["kind"] == "solve":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        n = nx * ny * nz
        m = (nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1) + nx * nz
        return {"bytes": 68.0 * n + 48.0 * m, "flops": m * (350.0 + 25.0 * case["iterations"])}
    n = _bodies(case)
    if case["kind"] == "frame":
        its = 70 if case["constants"] == "reference" else 10
        return {"bytes": n * (2 * 244.0 + 96.0), "flops": n * (3000.0 + 25.0 * (its - 10))}
    per = 500.0 + (500.0 if case["scene"] == "random" else 2500.0)
    if case["kind"] == "diff":
        return {"bytes": n * (96.0 + 28.0 + 100.0), "flops": case["steps"] * n * (per + 300.0)}
    return {"bytes": n * (96.0 + 28.0), "flops": case["steps"] * n * per}


# ---- 64 bits ---------------------------------------------------------------------------------


def exact(case, seed):
    """The contact solve in 64 bits. The stepping cases have no such value: which vertex a support
    map takes, which face an EPA ends on and which pairs touch are decided by the single-precision
    values themselves, and a 64-bit run of the method finds other contacts. They are defined bit for
    bit instead."""
    if case["kind"] != "solve":
        return None
    pos, vel, omg, mass, moi, pairs, ground, ncub = _pile(case, seed)
    f8 = lambda x: np.asarray(x, np.float64)
    g = f8(ground)
    m = len(pairs)
    sph_a = np.isin(pairs["Type"], (SF, SS))
    sph_b = np.isin(pairs["Type"], (CS, SS))
    on_floor = np.isin(pairs["Type"], (CF, SF))
    a = pairs["IndexA"] + ncub * sph_a
    b = np.where(on_floor, len(pos), pairs["IndexB"] + ncub * sph_b)
    P = np.concatenate([f8(pos), g[None, 0:3]])
    V = np.concatenate([f8(vel), g[None, 3:6]])
    W = np.concatenate([f8(omg), g[None, 6:9]])
    im = 1.0 / np.concatenate([f8(mass), g[9:10]])
    ii = 1.0 / np.concatenate([f8(moi), g[10:11]])
    dot = lambda x, y: (x * y).sum(-1)
    n = f8(pairs["N"])
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    z = np.zeros(m)
    # the tangent switch is decided in single precision, as the solve does
    t1 = np.where((n[:, 0].astype(np.float32) >= np.float32(0.57735))[:, None],
                  np.stack([n[:, 1], -n[:, 0], z], 1), np.stack([z, n[:, 2], -n[:, 1]], 1))
    t2 = np.cross(n, t1)
    r1, r2 = f8(pairs["PointA"]) - P[a], f8(pairs["PointB"]) - P[b]
    depth = dot((P[a] + r1) - (P[b] + r2), n)
    bias0 = -float(np.float32(0.3)) / float(DT) * depth
    dirs, ang1, ang2, mk = [n, t1, t2], [], [], []
    for d in dirs:
        c1, c2 = np.cross(r1, d), np.cross(r2, d)
        ang1.append(c1)
        ang2.append(c2)
        mk.append(1.0 / (im[a] + im[b] + (ii[a] * dot(c1, c1) - ii[b] * dot(c2, c2))))
    cr, mu = float(np.float32(0.2)), math.sqrt(2.0) * float(np.float32(0.5))
    for k in range(m):
        i, j = int(a[k]), int(b[k])
        rel = [float(dirs[q][k] @ (V[i] + np.cross(W[i], dirs[q][k]) - V[j] - np.cross(W[j], dirs[q][k])))
               for q in range(3)]
        bias = bias0[k] + cr * rel[0]
        ln, l1, l2 = (-rel[0] + bias) * mk[0][k], -rel[1] * mk[1][k], -rel[2] * mk[2][k]
        s = [0.0, 0.0, 0.0]
        dl = [0.0, 0.0, 0.0]
        for _ in range(case["iterations"]):
            old = s[0]
            s[0] = max(0.0, s[0] + ln)
            dl[0] = s[0] - old
            bound = mu * s[0]
            for q, x in ((1, l1), (2, l2)):
                old = s[q]
                s[q] = min(bound, max(-bound, s[q] + x))
                dl[q] = s[q] - old
        for q in range(3):
            V[i] += im[i] * dl[q] * dirs[q][k]
            W[i] += ii[i] * dl[q] * ang1[q][k]
            if j < len(pos):
                V[j] -= im[j] * dl[q] * dirs[q][k]
                W[j] -= ii[j] * dl[q] * ang2[q][k]
    return dict(velocity=torch.from_numpy(V[:-1].copy()), omega=torch.from_numpy(W[:-1].copy()))
