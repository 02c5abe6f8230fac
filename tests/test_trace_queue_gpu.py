"""The ray-cast queue at the sizes where its hand-out can go wrong, and the
quantized box test on ray forms it treats apart, against the same traversal
compiled for the host one ray at a time (hit ids and t, b1, b2 bit for bit;
the triangle arithmetic is the same on both sides and the closest hit does not
depend on the order of the tests)."""
import numpy as np
import pytest

import dort_b200 as db
from dort_b200 import scenes

torch = pytest.importorskip("torch")


def random_rays(n, seed):
    """Rays through the unit cube: finite and infinite ends, negative starts,
    axis-parallel directions of either sign."""
    rng = np.random.default_rng(seed)
    r = np.empty((n, 8), np.float32)
    r[:, 0:3] = rng.uniform(-0.5, 1.5, (n, 3))
    d = rng.normal(size=(n, 3))
    k = rng.integers(0, 6, n)
    axis = rng.integers(0, 3, n)
    sign = rng.choice([-1.0, 1.0], n)
    flat = k == 0
    d[flat] = 0.0
    d[flat, axis[flat]] = sign[flat]
    plane = k == 1
    d[plane, axis[plane]] = 0.0
    d[plane, (axis[plane] + 1) % 3] *= -1.0
    r[:, 4:7] = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    r[:, 3] = rng.choice([0.0, -0.7, 1e-3, 0.2], n)
    r[:, 7] = rng.choice([np.inf, 0.4, 2.0], n)
    return r


def cast(sc, rays, any_hit):
    n = len(rays)
    d = torch.from_numpy(rays).cuda()
    prim = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    tb = torch.zeros(n, 3, dtype=torch.float32, device="cuda")
    sc.raycast_device(d.data_ptr(), n, prim.data_ptr(), tb.data_ptr(), any_hit=any_hit)
    torch.cuda.synchronize()
    return prim.cpu().numpy().view(np.uint32), tb.cpu().numpy()


def warps_of(blocks_per_sm=8):
    return torch.cuda.get_device_properties(0).multi_processor_count * blocks_per_sm * 4


@pytest.mark.gpu
@pytest.mark.parametrize("watertight", [False, True])
def test_queue_sizes_against_host(watertight):
    verts, tris = scenes.random_triangles(3000, seed=3, sigma=0.05)
    w = warps_of()
    # a lone ray, part of a warp, one ray per warp, the shares where the first
    # chunk changes, the first sizes that use the cursor, several chunks
    sizes = sorted({1, 3, 31, 32, 33, w - 1, w, w + 1, 16 * w + 1, 64 * w, 64 * w + 1, 80 * w + 31})
    rays = random_rays(sizes[-1], 11)
    sc = db.Scene(verts, tris, watertight=watertight)
    ref, ref_tb, _ = db.host_check_raycast(verts, tris, rays, watertight=watertight)
    hit = ref != db.MISS
    assert hit.any() and not hit.all()
    for n in sizes:
        prim, tb = cast(sc, rays[:n], False)
        assert np.array_equal(prim, ref[:n]), n
        h = hit[:n]
        assert np.array_equal(tb[h].view(np.uint32), ref_tb[:n][h].view(np.uint32)), n
        assert not tb[~h].any()      # misses leave their t, b1, b2 alone
        occ, _ = cast(sc, rays[:n], True)
        assert np.array_equal(occ, h.astype(np.uint32)), n


@pytest.mark.gpu
@pytest.mark.parametrize("n_tris", [0, 1, 2, 3, 17])
def test_small_trees_against_host(n_tris):
    verts, tris = scenes.random_triangles(max(n_tris, 1), seed=n_tris, sigma=0.6)
    tris = tris[:n_tris]
    rays = random_rays(5000, 5)
    ref, ref_tb, _ = db.host_check_raycast(verts, tris, rays)
    sc = db.Scene(verts, tris)
    prim, tb = cast(sc, rays, False)
    assert np.array_equal(prim, ref)
    hit = ref != db.MISS
    assert np.array_equal(tb[hit].view(np.uint32), ref_tb[hit].view(np.uint32))


def test_boxes_never_cull_a_hit_on_the_host():
    """Closest hits through the tree equal the ones over all triangles (a tree
    whose root holds every triangle of a 2-triangle scene culls nothing else)."""
    verts, tris = scenes.random_triangles(400, seed=9, sigma=0.08)
    rays = random_rays(4000, 13)
    ref, ref_tb, _ = db.host_check_raycast(verts, tris, rays)
    best = np.full(len(rays), np.inf, np.float32)
    prim = np.full(len(rays), db.MISS, np.uint32)
    for k in range(len(tris)):
        p, tb, _ = db.host_check_raycast(verts, tris[k:k + 1], rays)
        hit = p != db.MISS
        better = hit & ((tb[:, 0] < best) | ((tb[:, 0] == best) & (prim != db.MISS)) |
                        (prim == db.MISS))
        best[better], prim[better] = tb[better, 0], k
    assert np.array_equal(prim, ref)
