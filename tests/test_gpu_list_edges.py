"""Exact results at the edges of the kernels' trips and tiles: the islands and colours of chains
whose manifold count lies around a block, a trip of several entries per thread and its remainder,
and the pair sort on keys that put whole warps, or all but one lane, on one digit."""
import ctypes

import numpy as np
import pytest

import beatbox as bb
from beatbox import scenes

pytestmark = pytest.mark.gpu


def chains(manifolds, length):
    """Rows of `length` spheres in contact (the last row holds the remaining manifolds)."""
    pos, rows = [], 0
    while manifolds:
        links = min(manifolds, length - 1)
        x = 0.99 * np.arange(links + 1)
        pos.append(np.stack([x, np.full_like(x, 3.0 * (rows // 96)), np.full_like(x, 3.0 * (rows % 96))], axis=1))
        manifolds -= links
        rows += 1
    pos = np.concatenate(pos)
    sb = scenes.SceneBuilder("physical")
    quat = np.tile(np.array([0.0, 0.0, 0.0, 1.0]), (len(pos), 1))
    sb.add(pos, quat, np.full((len(pos), 3), 0.5), scenes.SHAPE_SPHERE, scenes.BODY_DYNAMIC, 1.0, friction=0.5)
    sc = sb.build()
    sc["bounds"] = ([-8.0] * 3, [512.0] * 3)
    return sc, rows


@pytest.mark.parametrize("length", [2, 64])
@pytest.mark.parametrize("manifolds", [1, 31, 33, 511, 512, 513, 1536, 2047, 2049, 3073, 8193, 12289])
def test_chains_give_one_island_each_and_every_contact_a_colour(manifolds, length):
    sc, rows = chains(manifolds, length)
    p = bb.default_params()
    p.solver, p.quirks = bb.SOLVER_PGS_SOFT, bb.QUIRKS_PHYSICAL
    w = bb.world_from_scene(sc, params=p)
    for _ in range(2):  # the second step reuses the first one's colours
        w.step(1.0 / 240.0, 1)
        w.sync()
        st = w.stats()
        assert st["error_flags"] == 0
        assert st["manifold_count"] == manifolds
        assert st["island_count"] == rows
        assert st["graph_color_overflow"] == 0 and st["solved_manifolds"] == manifolds
    w.close()


def dptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("n", [31, 33, 8191, 8192, 8193, 3 * 8192 + 31])
@pytest.mark.parametrize("kind", ["constant", "two", "one_lane", "high_digit", "falling"])
def test_sort_ranks_of_crowded_digits(n, kind):
    import torch

    i = np.arange(n, dtype=np.uint32)
    keys = {"constant": np.full(n, 0xA5A5A5A5, np.uint32), "two": np.where(i % 3 == 0, 7, 0x01000007).astype(np.uint32),
            "one_lane": np.where(i % 32 == 17, 0, 0xFFFFFFFF).astype(np.uint32), "high_digit": (i % 5) << np.uint32(24),
            "falling": np.uint32(0xFFFFFFFF) - i}[kind].astype(np.uint32)
    kin, vin = (torch.from_numpy(a.view(np.int32).copy()).cuda() for a in (keys, i))
    kout, vout = torch.full_like(kin, -1), torch.full_like(vin, -1)
    torch.cuda.synchronize()
    assert bb.load_library().bb_radix_sort_pairs(dptr(kin), dptr(vin), dptr(kout), dptr(vout), n, 32, None) == bb.OK
    torch.cuda.synchronize()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(vout.cpu().numpy().view(np.uint32), order.astype(np.uint32))
    assert np.array_equal(kout.cpu().numpy().view(np.uint32), keys[order])
