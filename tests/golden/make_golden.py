"""Generates tests/golden/*.npz from the oracle.

The reference repository ships no golden vectors, so these fixtures are produced by the oracle
(the CPU restatement of the reference step) and pin it against unintended changes; the CUDA
library is compared with the same oracle in the GPU tests.  Re-run after a deliberate change to
the restated algorithm:  python tests/golden/make_golden.py

colour_sweeps.npz holds the library's own bits and is written only when it is named, on a machine
with a GPU:  python tests/golden/make_golden.py colour_sweeps
"""
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))
sys.path.insert(0, os.path.join(ROOT, "beat-box_b200"))
sys.path.insert(0, os.path.join(ROOT, "oracle"))

import pyoracle  # noqa: E402
from beatbox import scenes  # noqa: E402

CASES = {
    "grid_4x3": dict(scene=lambda: scenes.box_grid(n_side=4, layers=3), solver=1, quirks=0),
    "grid_4x3_reference": dict(scene=lambda: scenes.box_grid(n_side=4, layers=3, inertia="reference", density=5.0),
                               solver=1, quirks=7),
    "mixed_400_avbd": dict(scene=lambda: scenes.mixed_column(n_bodies=400, seed=5), solver=2, quirks=0),
}
STEPS = 20


def params(case, sc):
    p = pyoracle.default_params()
    p.solver, p.quirks = case["solver"], case["quirks"]
    p.iterations = p.relax_iterations = 8
    p.avbd_iterations = 4
    if sc.get("bounds") is not None:
        p.world_min[:] = sc["bounds"][0]
        p.world_extent[:] = sc["bounds"][1]
    return p


def read(o, code, dtype):
    cnt, buf = o.debug_read(code)
    return buf[: cnt * np.dtype(dtype).itemsize].view(dtype).copy()


def generate(name):
    case = CASES[name]
    sc = case["scene"]()
    o = pyoracle.Oracle(sc, params=params(case, sc))
    o.collide(2)
    out = dict(morton=read(o, 1, np.uint32), sorted_ids=read(o, 3, np.uint32), lbvh_child=read(o, 4, np.int32),
               pairs=read(o, 7, np.uint32))
    o = pyoracle.Oracle(sc, params=params(case, sc))
    traj = []
    for _ in range(STEPS):
        o.step(1 / 60, 4)
        traj.append(o.state()["pos"])
    out["trajectory"] = np.asarray(traj)
    out["final_stats"] = np.array([o.stats()[k] for k in ("manifold_count", "contact_count", "graph_color_count")])
    return out


def colour_sweeps():
    """Settled piles and the states one substep of the library makes of them."""
    sys.path.insert(0, os.path.dirname(HERE))
    import test_gpu_colour_sweeps as t

    piles = {n: t.settled_pile(pyoracle, n) for n in sorted({n for n, _ in t.CASES})}
    out = {f"settled_{k}_{n}": v for n, st in piles.items() for k, v in st.items()}
    for i, (n, kw) in enumerate(t.CASES):
        got, st = t.run_case(pyoracle, n, kw, piles[n])
        assert st["error_flags"] == 0
        out.update({f"{k}_{i}": v for k, v in got.items()})
    return out


def main():
    if "colour_sweeps" in sys.argv[1:]:
        np.savez_compressed(os.path.join(HERE, "colour_sweeps.npz"), **colour_sweeps())
        print("wrote colour_sweeps")
        return
    for name in CASES:
        np.savez_compressed(os.path.join(HERE, f"{name}.npz"), **generate(name))
        print("wrote", name)


if __name__ == "__main__":
    main()
