"""Performance cases of the rigid-body step library: the calls its users make, over their sizes.

Most cases are one frame of a host program that owns the state of its bodies: upload poses and
velocities from pinned host buffers (``World.write_state``), advance one step
(``World.step(dt, substeps)``), read poses and velocities back (``World.read_state``).  Every pass
starts from the same state, as a rollout from a checkpoint does, and the warm-start contacts are
those of the pass before.  The states are mid-run ones: a scene is rolled forward until its pile
has formed (or starts in contact, as the pyramids do) and every body is then jolted by a random
velocity, so that the bodies are awake and in contact.

The other cases are a device-resident world at rest (a level whose stacks have gone to sleep),
requests to the serving loop, and the device radix sort on its own.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "beat-box_b200"))

import beatbox as bb  # noqa: E402
from beatbox import reference_scenes, scenes  # noqa: E402

DT = 1.0 / 60.0
JOLT = 0.25  # m/s (and rad/s), above the sleep thresholds


def listed():
    return [
        # the smallest call: the reference's first demo scene (18 cubes on a floor) with its
        # default solver and parameters, one frame of an interactive viewer
        {"name": "demo_scene_avbd", "kind": "demo", "scene": 1},
        # the 1,000-box grid, a small game level: PGS_SOFT 8 + 8 iterations, 4 substeps
        {"name": "grid_1000_pgs", "kind": "pile", "solver": "pgs", "bodies": 1000, "spheres": 0.0, "iterations": 8,
         "substeps": 4},
        # a mid-size mixed pile under AVBD (the reference's default solver), default stiffness
        {"name": "pile_20k_avbd", "kind": "pile", "solver": "avbd", "bodies": 20000, "spheres": 0.4, "iterations": 10,
         "substeps": 4},
        # 100k boxes and spheres poured into a container: one deep pile, one island
        {"name": "column_100k_pgs", "kind": "column", "bodies": 100_000, "iterations": 10,
         "substeps": 4},
        # a million boxes in pyramids, all awake: the largest world
        {"name": "pyramids_1m_pgs", "kind": "pyramids", "pyramids": 1000, "iterations": 10, "substeps": 4},
        # a level at rest: every stack asleep, the transforms read for rendering
        {"name": "rest_200k", "kind": "rest", "pyramids": 200, "iterations": 10, "substeps": 4},
        # many independent worlds in one batch (training environments): sizes 16..2048
        {"name": "batch_1024_pgs", "kind": "batch", "solver": "pgs", "worlds": 1024, "iterations": 8, "substeps": 4},
        # the same kind of batch under AVBD, 4 iterations, one pass per step
        {"name": "batch_256_avbd", "kind": "batch", "solver": "avbd", "worlds": 256, "iterations": 4, "substeps": 1},
        # concave voxel bodies
        {"name": "voxel_5k_pgs", "kind": "voxel", "bodies": 5000, "iterations": 10, "substeps": 4},
        # serving: a burst of jobs, each a new world advanced a few steps and read back
        {"name": "served_12_jobs", "kind": "served", "jobs": 12, "largest": 4096, "steps": 4},
        # the device radix sort on its own, as a user's own pipeline calls it
        {"name": "sort_16m", "kind": "sort", "keys": 1 << 24, "bits": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["demo", "pile", "pile", "pile", "column", "pyramids", "rest", "batch", "voxel", "served", "sort"])
    if kind == "demo":  # the demo scenes of 17..1,001 bodies; the variant seeds the bodies' jolts
        return {"kind": kind, "scene": rng.choice([1, 2, 3, 4, 7]), "variant": rng.randrange(1, 1000)}
    if kind == "pile":
        solver = rng.choice(["pgs", "avbd"])
        return {"kind": kind, "solver": solver, "bodies": _log_int(rng, 100, 40_000 if solver == "pgs" else 20_000),
                "spheres": round(rng.uniform(0.0, 0.6), 2), "iterations": rng.randrange(4, 11),
                "substeps": rng.randrange(1, 5)}
    if kind == "column":
        return {"kind": kind, "bodies": _log_int(rng, 3000, 100_000), "iterations": rng.randrange(4, 11), "substeps": 4}
    if kind in ("pyramids", "rest"):
        return {"kind": kind, "pyramids": _log_int(rng, 2, 400 if kind == "pyramids" else 200),
                "iterations": rng.randrange(4, 11), "substeps": rng.randrange(1, 5)}
    if kind == "batch":
        solver = rng.choice(["pgs", "pgs", "avbd"])
        return {"kind": kind, "solver": solver, "worlds": _log_int(rng, 8, 1024 if solver == "pgs" else 256),
                "iterations": rng.randrange(4, 9), "substeps": rng.randrange(1, 5 if solver == "pgs" else 3)}
    if kind == "voxel":
        return {"kind": kind, "bodies": _log_int(rng, 60, 5000), "iterations": rng.randrange(4, 11),
                "substeps": rng.randrange(1, 5)}
    if kind == "served":
        return {"kind": kind, "jobs": rng.randrange(2, 13), "largest": _log_int(rng, 256, 4096),
                "steps": rng.randrange(1, 5)}
    return {"kind": "sort", "keys": _log_int(rng, 1000, 1 << 24), "bits": rng.choice([16, 24, 30, 32])}


# ---- scenes -----------------------------------------------------------------------------------
def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float32).pin_memory()
    out = t.numpy()
    out[...] = a
    return out


def _jolt(state, flags, seed):
    rng = np.random.default_rng(seed)
    dyn = (flags & bb.BODY_DYNAMIC) != 0
    for k in ("vel", "omega"):
        state[k][dyn] += rng.normal(0.0, JOLT, (int(dyn.sum()), 3)).astype(np.float32)


def _params(case):
    if case.get("solver") == "avbd":
        kw = dict(solver=bb.SOLVER_AVBD, avbd_iterations=int(case["iterations"]))
    else:
        kw = dict(solver=bb.SOLVER_PGS_SOFT, iterations=int(case["iterations"]),
                  relax_iterations=int(case["iterations"]))
    return bb.make_params(quirks=bb.QUIRKS_PHYSICAL, **kw)


def _frame_state(world, flags, seed, dt, substeps, settle):
    """Rolls the world `settle` steps, jolts its bodies; the host buffers of the frame loop."""
    for _ in range(settle):
        world.step(dt, substeps)
    world.sync()
    state = world.read_state()
    _jolt(state, flags, seed)
    return {"world": world, "in": {k: _pinned(v) for k, v in state.items()},
            "out": {k: _pinned(v) for k, v in state.items()}, "dt": dt, "substeps": substeps}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "demo":
        # the reference's manager: default solver (AVBD), default parameters, one pass per frame
        k = int(case["scene"])
        scene = reference_scenes.scene_2(seed=seed + int(case.get("variant", 0))) if k == 2 \
            else reference_scenes.reference_scene(k)
        m = bb.RigidBodyManager(int(scene["n"]), pairs_per_body=64 if "voxel_shapes" in scene else 16)
        m.create(iterations=5)
        m.world.add_scene(scene)
        for _ in range(90):
            m.simulate()
        st = _frame_state(m.world, scene["flags"], seed + 7919 * int(case.get("variant", 0)), m.TIME_STEP, 1, 0)
        st["manager"] = m
        return st
    if kind in ("pile", "column", "voxel", "pyramids", "rest"):
        if kind == "pile":
            scene = scenes.pile(int(case["bodies"]), seed=seed, sphere_fraction=float(case["spheres"]))
            settle = 40
        elif kind == "column":
            scene = scenes.mixed_column(int(case["bodies"]), seed=seed)
            settle = 290
        elif kind == "voxel":
            scene = scenes.voxel_pile(int(case["bodies"]), seed=seed)
            settle = 70
        else:
            # layers half a millimetre into each other: in contact from the first substep (the
            # boxes of a layer stay 1 mm apart)
            scene = scenes.pyramids(int(case["pyramids"]), seed=seed)
            y = scene["pos"][1:, 1]
            y[...] = 0.4995 + 0.9995 * np.round((y - 0.5) / 1.001)
            settle = 0
        world = bb.World(int(scene["n"]), pairs_per_body=64 if kind == "voxel" else 8 if kind == "pyramids" else 16)
        world.add_scene(scene)
        p = _params(case)
        if scene.get("bounds") is not None:
            p.world_min[:], p.world_extent[:] = scene["bounds"]
        world.set_params(p)
        if kind == "rest":  # until every stack sleeps
            for _ in range(60):
                world.step(DT, 4)
            world.sync()
            for _ in range(20):
                if world.stats()["sleeping_count"] == int(scene["n"]) - 1:
                    break
                for _ in range(10):
                    world.step(DT, 4)
            return {"world": world, "dt": DT, "substeps": int(case["substeps"])}
        return _frame_state(world, scene["flags"], seed, DT, int(case["substeps"]), settle)
    if kind == "batch":
        n_worlds = int(case["worlds"])
        n_templates = min(n_worlds, 64)  # piles of the batch, each used by several worlds
        sizes = scenes.batch_sizes(n_templates, seed=0)
        templates = [scenes.pile(int(n), seed=seed + k + 1) for k, n in enumerate(sizes)]
        use = [templates[k % n_templates] for k in range(n_worlds)]
        world = bb.World(sum(int(s["n"]) for s in use), pairs_per_body=8)
        for s in use:
            world.add_world(s, *s["bounds"])
        world.set_params(_params(case))
        flags = np.concatenate([s["flags"] for s in use])
        return _frame_state(world, flags, seed, DT, int(case["substeps"]), 40)
    if kind == "served":
        sizes = scenes.batch_sizes(int(case["jobs"]), seed=1, lo=64, hi=int(case["largest"]))
        jobs = [scenes.pile(int(n), seed=seed + k) for k, n in enumerate(sizes)]
        p = [bb.make_params(solver=bb.SOLVER_PGS_SOFT, iterations=10, relax_iterations=10, quirks=bb.QUIRKS_PHYSICAL),
             bb.make_params(solver=bb.SOLVER_AVBD, avbd_iterations=4, avbd_beta=10.0, quirks=bb.QUIRKS_PHYSICAL)]
        for s in jobs:  # a job starts in motion, its bodies in contact at their corners
            _jolt(s, s["flags"], seed)
        state = {"server": bb.Server(hbm_budget_bytes=3 << 30, max_active=64, pairs_per_body=16), "jobs": jobs,
                 "arrays": [bb.scene_request_arrays(s) for s in jobs], "params": p, "steps": int(case["steps"]), "next": 0}
        for _ in range(6):  # until the slots of the batches are in use, as in a server that has run for a while
            run(state)
            if state["server"].stats()["evictions"]:
                break
        return state
    n, bits = int(case["keys"]), int(case["bits"])
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    keys = torch.randint(0, 1 << min(bits, 31), (n,), device="cuda", dtype=torch.int64, generator=g)
    if bits == 32:
        keys = keys * 2 + torch.randint(0, 2, (n,), device="cuda", dtype=torch.int64, generator=g) - (1 << 31)
    keys = keys.to(torch.int32)
    vals = torch.arange(n, device="cuda", dtype=torch.int32)
    return {"keys": keys, "vals": vals, "keys_out": torch.empty_like(keys), "vals_out": torch.empty_like(vals),
            "n": n, "bits": bits}


# ---- passes ------------------------------------------------------------------------------------
def run(state):
    if "in" in state:  # one frame: upload, step, read back
        w, s = state["world"], state["in"]
        w.write_state(s["pos"], s["quat"], s["vel"], s["omega"])
        if "manager" in state:
            state["manager"].simulate()
        else:
            w.step(state["dt"], state["substeps"])
        return w.read_state(state["out"])
    if "world" in state:  # the world lives on the device; the transforms go to the renderer
        state["world"].step(state["dt"], state["substeps"])
        return state["world"].read_transforms()
    if "server" in state:
        srv, first = state["server"], state["next"]
        state["next"] += len(state["jobs"])
        tickets = [srv.submit(first + k, state["steps"], state["params"][k % 2], DT, 4, scene=s, arrays=state["arrays"][k])
                   for k, s in enumerate(state["jobs"])]
        for t in tickets:
            r = srv.wait(t)
            if r["result"] != bb.OK:
                raise bb.BeatboxError(r["result"], f"a served job failed: {r}")
        return [srv.read_state(first + k, int(s["n"])) for k, s in enumerate(state["jobs"])]
    L = bb.load_library()
    bb._check(L.bb_radix_sort_pairs(state["keys"].data_ptr(), state["vals"].data_ptr(), state["keys_out"].data_ptr(),
                                    state["vals_out"].data_ptr(), state["n"], state["bits"],
                                    torch.cuda.current_stream().cuda_stream))
    return [state["keys_out"], state["vals_out"]]


# ---- the work of a pass --------------------------------------------------------------------------
def work(case):
    """Bytes: body state and properties once in and once out (64 + 48 B read, 64 B written), the
    persistent contacts once in and once out (64 B per contact, 32 B per manifold each way), the
    sort's keys and values once each way.  Operations: about 3 rows of 60 operations per contact and
    sweep, 2,000 per manifold and substep for the narrow phase.  Contacts per body are typical ones
    of the kind of scene."""
    kind = case["kind"]
    if kind == "sort":
        return {"bytes": 16.0 * case["keys"], "flops": 0.0}
    if kind == "rest":  # nothing moves: flags and timers, and the transforms of every body
        n = 1000.0 * case["pyramids"]
        return {"bytes": n * (8 + 32 + 48), "flops": 40.0 * n}
    sub, steps, manifolds, contacts = float(case.get("substeps", 1)), 1.0, 2.0, 6.0  # per body
    iterations = 2.0 * case.get("iterations", 10)
    if kind == "demo":
        n = {1: 19, 2: 1001, 3: 27, 4: 17, 7: 438}.get(int(case["scene"]), 100)
    elif kind == "pyramids":
        n, manifolds, contacts = 1000.0 * case["pyramids"], 3.0, 12.0
    elif kind == "batch":
        n = 420.0 * case["worlds"]
    elif kind == "served":
        n, sub, steps, iterations = case["largest"] / math.log(case["largest"] / 64.0) * case["jobs"], 4.0, float(case["steps"]), 20.0
    else:
        n = float(case["bodies"])
        if kind == "column":
            manifolds, contacts = 1.5, 3.0
    nbytes = n * (64 + 48 + 64) + 2 * n * (32 * manifolds + 64 * contacts)
    return {"bytes": steps * nbytes, "flops": steps * sub * n * (180.0 * contacts * iterations + 2000.0 * manifolds)}


def exact(case, seed):
    """The sort's answer from torch's stable sort.  A step has none here: its contact decisions,
    colour order and sweeps are a pipeline of their own, and one that is restated in 64 bits is the
    oracle of this repository's tests."""
    if case["kind"] != "sort":
        return None
    s = prepare(case, seed)
    bits = s["bits"]
    order = torch.sort(s["keys"].to(torch.int64) & ((1 << bits) - 1 if bits < 32 else 0xFFFFFFFF), stable=True).indices
    return [s["keys"][order], s["vals"][order]]
