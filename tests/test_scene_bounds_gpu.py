"""The scene's bounds, which a device-built scene takes from the mesh scan's
threads: light from an environment starts on a disk around them, so the light
tracer's image shows them.  The vertices that decide them lie in the first, a
middle and the last thread's share, or all in one."""
import numpy as np
import pytest

import dort_b200 as db
from dort_b200 import scenes

N = 8 * 32768 + 29     # eight threads' shares, the last ones ragged


@pytest.mark.gpu
@pytest.mark.parametrize("at", [(0, N // 2, N - 1), (N - 1,), (3 * 32768 + 7,)])
def test_bounds_of_the_device_build_are_the_hosts(cuda, at):
    sd = scenes.env_test_scene()
    verts, tris = scenes.random_triangles(N - len(sd["tris"]), seed=6, sigma=0.005)
    verts = np.concatenate([sd["verts"], 0.5 * verts]).astype(np.float32)
    tris = np.concatenate([sd["tris"], tris + len(sd["verts"])]).astype(np.uint32)
    tris = np.roll(tris, N // 3, axis=0)
    mat = np.roll(np.concatenate([sd["tri_material"], np.zeros(N - len(sd["tris"]), np.uint32)]),
                  N // 3)
    far = [(9.0, 0.5, 1.0), (-2.0, 7.0, -8.0), (1.0, -1.0, 11.0)]
    for k, t in enumerate(at):
        # a sliver out to a corner of its own
        first = len(verts)
        verts = np.concatenate([verts, np.array([far[k]], np.float32) +
                                np.array([[0, 0, 0], [0.01, 0, 0], [0, 0.01, 0]], np.float32)])
        tris[t] = (first, first + 1, first + 2)
    sd.update(verts=verts.astype(np.float32), tris=tris, tri_material=mat.astype(np.uint32))
    p = db.render_params(sd["camera"], 48, 32, 64, max_depth=3, seed=4, renderer="lt")
    img = [db.scene_from_dict(sd, bvh_build=b).render(p)[0] for b in ("device", "host")]
    assert img[1].mean() > 0
    # the same paths; splats add in any order
    np.testing.assert_allclose(img[0], img[1], rtol=1e-4, atol=1e-5 * img[1].max())
