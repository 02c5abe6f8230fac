"""Rays that meet no box by their form (an origin at infinity or beyond what
distances can be computed from, an empty interval, no position at all) miss,
and cost the host-compiled traversal no more than ordinary ones do (a walk of
the whole tree, which lets such a ray's boxes pass, takes a thousand times as
long)."""
import numpy as np
import pytest

import dort_b200 as db
from dort_b200 import scenes
from tests.test_box_margin import SLOWER, timed

COUNT = 400


def ordinary(seed=1):
    rng = np.random.default_rng(seed)
    rays = np.zeros((COUNT, 8), np.float32)
    p = rng.uniform(0.2, 0.8, (COUNT, 3))
    o = rng.uniform(-0.5, 1.5, (COUNT, 3))
    rays[:, 0:3] = o
    rays[:, 4:7] = (p - o) / np.linalg.norm(p - o, axis=1, keepdims=True)
    rays[:, 7] = np.inf
    return rays


def forms():
    out = {}
    for far in (np.inf, 3e38, 1e30, 1e19):
        for axes in ([0], [0, 2], [1]):
            r = ordinary()
            r[:, axes] = far
            r[:, 4 + axes[0]] = 0          # 1e20 as a reciprocal
            out[f"origin {far} on {axes}"] = r
        r = ordinary()
        r[:, 0:3] = far
        r[:, 4:7] = 0
        out[f"origin {far}, no direction"] = r
    for lo, hi in ((0.0, -1.0), (1e-3, 0.0), (0.5, 0.4), (0.0, -np.inf)):
        r = ordinary()
        r[:, 3], r[:, 7] = lo, hi
        out[f"interval {lo} to {hi}"] = r
    r = ordinary()
    r[:, 0:7] = np.nan
    out["nothing defined"] = r
    return out


def test_rays_that_meet_no_box_end_at_once():
    verts, tris = scenes.random_triangles(60000, seed=2, sigma=0.02)
    base, (prim, _, _) = timed(verts, tris, ordinary())
    assert (prim != db.MISS).mean() > 0.9
    for name, rays in forms().items():
        took, (prim, _, _) = timed(verts, tris, rays)
        assert (prim == db.MISS).all(), name
        assert took < SLOWER * base + 0.1, (name, took, base)


@pytest.mark.gpu
@pytest.mark.parametrize("watertight", [False, True])
@pytest.mark.parametrize("any_hit", [False, True])
def test_forms_on_the_device(cuda, watertight, any_hit):
    """The same rays, an ordinary one after every other, through the device's
    queue: the odd ones miss, the ordinary ones keep their hits."""
    verts, tris = scenes.random_triangles(60000, seed=2, sigma=0.02)
    sc = db.Scene(verts, tris, watertight=watertight)
    ref, _, _ = db.host_check_raycast(verts, tris, ordinary(), watertight=watertight)
    for name, rays in forms().items():
        both = np.empty((2 * COUNT, 8), np.float32)
        both[0::2], both[1::2] = rays, ordinary()
        if any_hit:
            got = sc.raycast(both, any_hit=True)
            assert not got[0::2].any(), name
            assert np.array_equal(got[1::2] != 0, ref != db.MISS), name
        else:
            got, _ = sc.raycast(both)
            assert (got[0::2] == db.MISS).all(), name
            assert np.array_equal(got[1::2], ref), name
