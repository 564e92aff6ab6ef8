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


# ---- against the FP64 oracle on the GPU's own contacts --------------------------------------------
# The oracle takes the geometry that the GPU's narrow phase made (so no contact decision differs),
# colours it itself and runs the colours one after the other.  Rounding leaves the oracle's own FP32
# build within 3e-6 m/s and 6e-6 rad/s of its FP64 build on these scenes; another order of the
# colours moves 1 % of the bodies by 7e-3 m/s and more.  The bounds lie between: 1e-4 of the value + 2e-5
# m/s, 4e-5 rad/s (a box's half extent is 0.5 m), 1e-6 m.
REL, FLOORS = 1e-4, dict(pos=1e-6, vel=2e-5, omega=4e-5)


def jolted(sc, seed=0):
    rng = np.random.default_rng(seed)
    dyn = (sc["flags"] & bb.BODY_DYNAMIC) != 0
    for k in ("vel", "omega"):
        sc[k][dyn] += rng.normal(0.0, 0.25, (int(dyn.sum()), 3)).astype(np.float32)
    return sc


def tray(m):
    """m x m yawed boxes on one dynamic plate: a body with more manifolds than there are colours."""
    sb = scenes.SceneBuilder("physical")
    sb.add_static_box([0, -50, 0], [50, 50, 50])
    half, i = 0.55 * m + 1.0, np.arange(m * m)
    fl = scenes.BODY_DYNAMIC | scenes.BODY_GRAVITY
    sb.add([[0, 0.499, 0]], [[0, 0, 0, 1.0]], [[half, 0.5, half]], scenes.SHAPE_BOX, fl, 4000.0 * half * half)
    pos = np.stack([(i % m - (m - 1) / 2) * 1.1, np.full(m * m, 1.498), (i // m - (m - 1) / 2) * 1.1], axis=1)
    sb.add(pos, scenes.yaw_rotations(scenes.uniform(3, 1, m * m, 0, 6.28)), np.full((m * m, 3), 0.5), scenes.SHAPE_BOX,
           fl, 1000.0)
    sc = sb.build()
    sc["bounds"] = ([-64.0] * 3, [128.0] * 3)
    return jolted(sc)


def follows_the_oracle(po, sc, p, substeps=2):
    """Steps both through `substeps` (the second one starts with the first one's impulses)."""
    w = bb.world_from_scene(sc, params=p)
    o = po.Oracle(sc, params=p, threads=os.cpu_count() or 1)
    for _ in range(substeps):
        w.step(DT / 4, 1)
        w.sync()
        man, con = w.debug_read("manifolds"), w.debug_read("contacts")
        o.inject_manifolds(man, con)
        o.step(DT / 4, 1)
        cnt, buf = o.debug_read(10)
        assert np.array_equal(man["color"], buf[:4 * cnt].view(np.uint32))
        g, r = w.read_state(), o.state()
        for k, floor in FLOORS.items():
            over = np.abs(g[k] - r[k]) - (REL * np.abs(r[k]) + floor)
            assert over.max() <= 0.0, (k, over.max())
    st = w.stats()
    w.close()
    assert st["error_flags"] == 0
    return st, man


@pytest.mark.parametrize("m", [6, 8, 12])  # 5, 33 and 113 manifolds left to the overflow bucket
def test_a_body_with_more_manifolds_than_colours(oracle_lib, m):
    sc = tray(m)
    st, _ = follows_the_oracle(oracle_lib, sc, params(oracle_lib, sc))
    assert st["graph_color_overflow"] == m * m + 1 - 32
