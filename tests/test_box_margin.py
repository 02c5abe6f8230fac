"""The box test against the triangle test alone: rays aimed at the edges and
vertices of meshes at the coordinate origin, away from it and in a much larger
scene, from one to a thousand mesh sizes away, hit what the oracle's test of
every triangle without any box (the same operations, each rounded on its own)
hits.  There the triangle test reports hits that pass the triangle, and the
box around it, by its own rounding, which grows with the distance.

Not compared: rays within 0.02 of parallel to the triangle that either side
found.  Their distance is off by 50 times the rounding and more, so the order
of two triangles' distances is not defined in 32 bits."""
import time

import numpy as np
import pytest

import dort_b200 as db
from oracle import pyoracle as po
from tests.raycheck import classify

SIZE = 0.04
SLANT = 0.02


def grid(n, size, bump, rng):
    """n x n quads on the x-z plane around the origin, heights +- bump / 2 of a quad."""
    x = np.linspace(-size / 2, size / 2, n + 1)
    gx, gz = np.meshgrid(x, x, indexing="ij")
    y = rng.uniform(-0.5, 0.5, gx.shape) * bump * size / n
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    a = (i * (n + 1) + j).ravel()
    t = np.concatenate([np.stack([a, a + 1, a + n + 2], 1), np.stack([a, a + n + 2, a + n + 1], 1)])
    return np.stack([gx, y, gz], -1).reshape(-1, 3), t


def mesh(kind, where, rng):
    """A mesh of 32 x 32 quads, and in a scene a ground 500 times its size."""
    v, t = grid(32, SIZE, {"flat": 0.0, "bumpy": 0.6}[kind], rng)
    aimed = len(t)
    if where == "scene":
        ground, tg = grid(2, 500 * SIZE, 0.0, rng)
        t = np.concatenate([t, tg + len(v)])
        v = np.concatenate([v, ground - [0, 0.1, 0]])
    v = v + {"offset": (1, 0, 1), "far": (100, 0, 50)}.get(where, (0, 0, 0))
    return v.astype(np.float32), t.astype(np.uint32), aimed


def edge_rays(verts, tris, n, sizes, rng):
    """Rays at points of edges (a fifth at vertices) from `sizes` mesh sizes
    away; half of them with a zero x or z direction."""
    v = verts.astype(np.float64)
    tri = v[tris[rng.integers(0, len(tris), n)]]
    k, i = np.arange(n), rng.integers(0, 3, n)
    u = rng.uniform(0, 1, (n, 1)) * (rng.random((n, 1)) < 0.8)
    p = tri[k, i] + u * (tri[k, (i + 1) % 3] - tri[k, i])
    d = rng.normal(size=(n, 3))
    zero = np.where(rng.random(n) < 0.5, 2 * rng.integers(0, 2, n), -1)
    for a in (0, 2):
        d[zero == a, a] = 0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = (p - d * sizes * SIZE).astype(np.float32)
    d = p - o
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = o
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    for a in (0, 2):
        rays[zero == a, 4 + a] = 0
    rays[:, 7] = np.inf
    return rays


def slant(verts, tris, prim, rays):
    hit = prim != db.MISS
    t = verts.astype(np.float64)[tris[np.where(hit, prim, 0)]]
    nn = np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    c = np.abs((nn * rays[:, 4:7]).sum(1)) / np.linalg.norm(nn, axis=1)
    return np.where(hit, c, 1.0)


@pytest.mark.parametrize("where", ["origin", "offset", "far", "scene"])
@pytest.mark.parametrize("kind,sizes,count", [("flat", 1, 10000), ("flat", 1000, 100000),
                                              ("bumpy", 1, 10000), ("bumpy", 30, 10000),
                                              ("bumpy", 1000, 100000)])
def test_no_hit_is_culled(kind, where, sizes, count):
    rng = np.random.default_rng(sizes)
    verts, tris, aimed = mesh(kind, where, rng)
    rays = edge_rays(verts, tris[:aimed], count, sizes, rng)
    ref, ref_tb = po.brute_raycast(verts, tris, rays)
    got, tb, _ = db.host_check_raycast(verts, tris, rays)
    assert (ref != db.MISS).sum() > count // 3
    clear = np.minimum(slant(verts, tris, ref, rays), slant(verts, tris, got, rays)) > SLANT
    assert clear.mean() > 0.9
    _, _, nearer, bugs = classify(verts, tris, rays[clear], got[clear], tb[clear], ref[clear],
                                  ref_tb[clear])
    assert bugs == [] and nearer == []


# A ray from far away visits up to 10 times the nodes of one from near by; a
# walk of the whole tree visits 1,000 times as many and more.
SLOWER = 60


def timed(verts, tris, rays):
    """Seconds of the traversal alone (the build's are taken off) and results."""
    best = []
    for r in (rays, rays[:0]):
        took = []
        for _ in range(3):
            t = time.perf_counter()
            got = db.host_check_raycast(verts, tris, r)
            took.append(time.perf_counter() - t)
            if r is rays:
                res = got
        best.append(min(took))
    return max(best[0] - best[1], 0.0), res


@pytest.mark.parametrize("sizes", [100, 10000])
def test_rays_from_far_away_do_not_visit_the_whole_tree(sizes):
    """The margin is bounded by the nodes' own size."""
    verts, tris = grid(200, 1.0, 0.6, np.random.default_rng(4))
    verts, tris = verts.astype(np.float32), tris.astype(np.uint32)

    def aimed(dist):
        rng = np.random.default_rng(5)
        rays = np.zeros((400, 8), np.float32)
        p = verts[rng.integers(0, len(verts), 400)].astype(np.float64)
        d = rng.normal(size=(400, 3))
        d[:, 1] = np.abs(d[:, 1]) + 0.5
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        o = (p + d * dist).astype(np.float32)
        rays[:, 0:3] = o
        rays[:, 4:7] = (p - o) / np.linalg.norm(p - o, axis=1, keepdims=True)
        rays[:, 7] = np.inf
        return rays

    base, _ = timed(verts, tris, aimed(1.0))
    took, _ = timed(verts, tris, aimed(float(sizes)))
    assert took < SLOWER * base + 0.1, (took, base)


@pytest.mark.gpu
def test_tree_of_a_mesh_away_from_the_origin_is_as_good(cuda):
    """The boxes hold nothing that depends on where the node is: moved away
    from the coordinate origin, a mesh builds as good a tree, up to its
    vertices' rounding there (quads of 0.06 at coordinates up to 102, whose
    floats are 8e-6 apart)."""
    v, t = grid(64, 4.0, 0.6, np.random.default_rng(3))
    cost = []
    for off in ((0, 0, 0), (100, 0, 50)):
        sc = db.Scene((v + np.array(off)).astype(np.float32), t.astype(np.uint32))
        cost.append(sc.bvh_cost()["sah"])
    assert abs(cost[1] / cost[0] - 1) < 0.05
