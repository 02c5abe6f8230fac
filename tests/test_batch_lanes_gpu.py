"""Batches of so many tiny jobs that the rays of one warp, and the last few
that its lanes share (eight lanes to a ray), belong to several scenes: every
job's image is the one the scene renders alone."""
import numpy as np
import pytest

import dort_b200 as db
from dort_b200 import scenes
from tests import ptcheck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jobs,spp", [(64, 8), (600, 20)])
def test_warps_of_several_scenes(cuda, jobs, spp):
    # one-pixel jobs, neighbours in other scenes; 600 x 20 paths are two or
    # three to a warp of the whole chip, 64 x 8 fewer than one
    kinds = [scenes.soup_with_light(int(n), k) for k, n in enumerate(np.geomspace(200, 8000, 12))]
    kinds += [scenes.cornell_variant("delt"), scenes.env_test_scene()]
    built = [db.scene_from_dict(sd) for sd in kinds]
    held = []
    for j in range(jobs):
        k = j % len(kinds)
        held.append((built[k], db.render_params(kinds[k]["camera"], 1, 1, spp, max_depth=6,
                                                seed=1000 + j)))
    b = db.Batch(held)
    b.render()
    assert b.stats()["error"] == 0
    got = np.concatenate([b.image(j) for j in range(jobs)])
    want = np.concatenate([sc.render(p)[0] for sc, p in held])
    assert (want.sum(axis=-1) > 0).mean() > 0.5
    # 12,000 paths: the odd one takes another branch in the other kernel
    assert ptcheck.forked_pixels(got, want) <= 2
    b.close()
