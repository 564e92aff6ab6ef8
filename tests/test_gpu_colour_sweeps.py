"""The PGS_SOFT colour sweeps give the bits that a serial order of the colours gives, where the
kernel's paths differ: no colouring rounds (every manifold in the serial overflow bucket), one or
two rounds (some), all coloured; single bodies and pairs (one tile, one warp); sweeps, impulse
accumulation, friction and integration switched off.  One substep from a settled pile; the
expected states (tests/golden/colour_sweeps.npz) were written by the kernel that this one
replaced, which ran the colours one after the other with a grid barrier between them."""
import os

import numpy as np
import pytest

import beatbox as bb
from beatbox import scenes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def params(po, sc, **kw):
    p = po.default_params()
    p.solver, p.quirks = bb.SOLVER_PGS_SOFT, bb.QUIRKS_PHYSICAL
    for k, v in kw.items():
        setattr(p, k, v)
    if sc.get("bounds") is not None:
        p.world_min[:] = sc["bounds"][0]
        p.world_extent[:] = sc["bounds"][1]
    return p


def settled_pile(po, n, seed=4):
    sc = dict(scenes.pile(n, seed=seed, sphere_fraction=0.3))
    o = po.Oracle(sc, params=params(po, sc))
    for _ in range(35):
        o.step(DT, 4)
    st = o.state()
    sc.update({k: st[k].astype(np.float32) for k in ("pos", "quat", "vel", "omega")})
    return sc


ALL = bb.SIM_DEFAULT_FLAGS
CASES = [  # bodies, parameters
    (60, dict(gc_rounds=0)), (60, dict(gc_rounds=1)), (60, dict(gc_rounds=2)), (60, dict(gc_rounds=32)),
    (1, {}), (2, {}), (33, {}), (250, {}), (600, dict(iterations=1, relax_iterations=0)),
    (60, dict(iterations=0, relax_iterations=3)), (60, dict(flags=ALL & ~bb.SIM_ADVECTION)),
    (60, dict(flags=ALL & ~bb.SIM_ACCUM_IMPULSE)), (60, dict(flags=ALL & ~bb.SIM_FRICTION)),
    (60, dict(flags=ALL & ~bb.SIM_ACCUM_IMPULSE, gc_rounds=1)),
]


GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "colour_sweeps.npz")


def run_case(po, n, kw):
    sc = settled_pile(po, n)
    w = bb.world_from_scene(sc, params=params(po, sc, **kw))
    w.step(DT / 4, 1)
    w.sync()
    return w.read_state(), w.stats()


@pytest.mark.parametrize("i", range(len(CASES)))
def test_one_substep_gives_the_serial_colour_order(oracle_lib, i):
    n, kw = CASES[i]
    got, st = run_case(oracle_lib, n, kw)
    assert st["error_flags"] == 0 and st["solved_manifolds"] == st["manifold_count"]
    assert (st["graph_color_overflow"] > 0) == (kw.get("gc_rounds", 32) < 3 and n > 2)
    with np.load(GOLDEN) as z:
        for k in got:
            assert np.array_equal(got[k], z[f"{k}_{i}"]), k
