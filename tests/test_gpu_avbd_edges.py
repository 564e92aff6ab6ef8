"""AVBD at the edges of its body lists: one support layer, as many as there are buckets for (64 layers x
32 colours, keys of two digits), towers and piles deeper than the layers; no post-stabilisation
sweeps, one, and several; buckets of less and of more than one block's bodies.  One substep; the FP64
oracle solves the GPU's contacts.

On these scenes rounding leaves the oracle's own FP32 build within 4.2e-6 m, 1.1e-3 m/s (a velocity is a
difference of positions, rounded to 2e-6 m at 40 m, over 1/240 s) and 8e-4 rad/s of its FP64 build;
another number of layers or sweeps moves some body by 6e-4 m or more.  The bounds lie between: 4e-5 m,
5e-3 m/s, 5e-3 rad/s."""
import numpy as np
import pytest

import beatbox as bb
from beatbox import scenes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
BOUNDS = dict(pos=4e-5, vel=5e-3, omega=5e-3)
NO_DEPTH = 0xFFFFFFFF
HEIGHTS = (1, 2, 3, 11, 12, 13, 20, 40)
EDGES = [(1, 4), (2, 1), (12, 0), (12, 1), (12, 8), (64, 1), (64, 4)]  # layers, post-stabilisation sweeps


def towers():
    sb = scenes.SceneBuilder("physical")
    sb.add_static_box([0, -50, 0], [50, 50, 50])
    pos = [[3.0 * t - 10.0, 0.497 + 0.997 * k, 0.0] for t, h in enumerate(HEIGHTS) for k in range(h)]
    pos.append([0.0, 10.0, 20.0])  # touches nothing: no depth
    n = len(pos)
    sb.add(pos, scenes.yaw_rotations(scenes.uniform(3, 1, n, 0, 6.28)), np.full((n, 3), 0.5), scenes.SHAPE_BOX,
           scenes.BODY_DYNAMIC | scenes.BODY_GRAVITY, 5.0)
    sc = sb.build()
    rng = np.random.default_rng(1)
    sc["vel"][1:] += rng.normal(0.0, 0.05, (n, 3)).astype(np.float32)
    sc["omega"][1:] += rng.normal(0.0, 0.05, (n, 3)).astype(np.float32)
    sc["bounds"] = ([-64.0] * 3, [128.0] * 3)
    return sc


def params(po, sc, layers, sweeps):
    p = po.default_params()
    p.solver, p.quirks, p.avbd_iterations = bb.SOLVER_AVBD, bb.QUIRKS_PHYSICAL, 4
    p.avbd_shock_layers, p.avbd_post_stab_sweeps = layers, sweeps
    p.avbd_k_min = 1e6  # stiff from the first substep, so that the order of the bodies counts
    p.world_min[:], p.world_extent[:] = sc["bounds"]
    return p


def read(o, code, dtype=np.uint32):
    cnt, buf = o.debug_read(code)
    return buf[: cnt * np.dtype(dtype).itemsize].view(dtype).copy()


def settled_pile(po):
    """2,000 boxes and spheres that PGS_SOFT rolled for 35 steps on the GPU."""
    sc = scenes.pile(2000, seed=4, sphere_fraction=0.3, density=5.0)
    p = params(po, sc, 12, 4)
    p.solver = bb.SOLVER_PGS_SOFT
    w = bb.world_from_scene(sc, params=p)
    for _ in range(35):
        w.step(DT, 4)
    st = w.read_state()
    w.close()
    return dict(sc, **{k: np.ascontiguousarray(v, np.float32) for k, v in st.items()})


@pytest.mark.parametrize("scene", ["towers", "pile"])
@pytest.mark.parametrize("layers,sweeps", EDGES)
def test_avbd_follows_the_oracle(oracle_lib, scene, layers, sweeps):
    sc = towers() if scene == "towers" else settled_pile(oracle_lib)
    p = params(oracle_lib, sc, layers, sweeps)
    w = bb.world_from_scene(sc, params=p)
    w.step(DT / 4, 1)
    w.sync()
    assert w.stats()["error_flags"] == 0 and w.stats()["avbd_violations"] == 0
    o = oracle_lib.Oracle(sc, params=p)
    o.inject_manifolds(w.debug_read("manifolds"), w.debug_read("contacts"))
    o.step(DT / 4, 1)
    assert np.array_equal(w.debug_read("body_colors"), read(o, 11))
    depth, want = w.debug_read("support_depth"), read(o, 13)
    # (a pass may hand depths on further than one layer; the cascade takes them up to the last layer)
    assert np.array_equal(np.minimum(depth, layers - 1), np.minimum(want, layers - 1))
    if scene == "towers":  # below 64 layers nothing cuts the towers off
        assert layers != 64 or (want[want != NO_DEPTH].max() == max(HEIGHTS) and np.array_equal(depth, want))
    g, r = w.read_state(), o.state()
    for k, bound in BOUNDS.items():
        err = np.abs(g[k] - r[k]).max()
        assert err <= bound, (k, err)
