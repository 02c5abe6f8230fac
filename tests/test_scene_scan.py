"""Scene creation's mesh scan (several threads on large meshes) refuses the
meshes the host build refuses, with the same message, wherever the fault is,
and finds the same bounds."""
import numpy as np
import pytest

import dort_b200 as db
from dort_b200 import scenes

N = 4 * 32768 + 17     # several threads' shares, the last one ragged


@pytest.mark.gpu
@pytest.mark.parametrize("at", [0, 32768, 2 * 32768 + 5, N - 1])
@pytest.mark.parametrize("fault", ["index", "nan", "large"])
def test_faults_are_refused_with_the_host_message(at, fault):
    verts, tris = scenes.random_triangles(N, seed=2)
    if fault == "index":
        tris = tris.copy()
        tris[at, 1] = len(verts)
    else:
        verts[3 * at + 2, 1] = np.nan if fault == "nan" else 2e15
    with pytest.raises(db.DortError) as dev:
        db.Scene(verts, tris)
    with pytest.raises(db.DortError) as host:
        db.Scene(verts, tris, bvh_build="host")
    assert str(dev.value) == str(host.value)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 32767, N])
def test_shading_records_of_both_builds_render_alike(n):
    """Device-made and host-made shading records, materials and light indices
    give the same image (one emissive triangle among materials of two kinds)."""
    sd = scenes.soup_with_light(n, 3)
    sd["materials"] = sd["materials"] + [{"kind": db.MAT_MIRROR, "color": (0.9, 0.8, 0.7)}]
    sd["tri_material"][: n // 2] = 2
    p = db.render_params(sd["camera"], 40, 30, 4, max_depth=4, seed=1)
    img = [db.scene_from_dict(sd, bvh_build=b).render(p)[0] for b in ("device", "host")]
    assert np.array_equal(img[0], img[1])
