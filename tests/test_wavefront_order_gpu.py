"""Deterministic frames add a path's direct-lighting terms in a fixed order:
the light strategy's before the BSDF strategy's, whatever the scheduling of
the stages.  Large frames of glossy surfaces under an area light, where many
vertices have an unblocked entry of each (with the two queues traced side by
side, some of these frames' pixels differ from one rendering to the next)."""
import numpy as np
import pytest

import dort_b200 as db
from dort_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity", [None, 1 << 16])
def test_deterministic_frames_repeat_to_the_bit(cuda, capacity):
    sd = scenes.cornell_variant("glos")
    sc = db.scene_from_dict(sd)
    p = db.render_params(sd["camera"], 512, 512, 16, max_depth=6, seed=3)
    tuning = {"deterministic": True}
    ref, _ = sc.render_wavefront(p, tuning)
    if capacity:
        tuning["queue_capacity"] = capacity
    for _ in range(6):
        img, _ = sc.render_wavefront(p, tuning)
        assert np.array_equal(img.view(np.uint32), ref.view(np.uint32))


def test_adjoint_forward_repeats_to_the_bit(cuda):
    sd = scenes.adjoint_scene(20000, seed=5)
    sc = db.scene_from_dict(sd)
    p = db.render_params(sd["camera"], 384, 384, 16, max_depth=6, seed=7)
    alb, em = sd["tri_albedo"], sd["tri_emission"]
    ref = sc.adjoint_forward(p, alb, em)
    for _ in range(6):
        img = sc.adjoint_forward(p, alb, em)
        assert np.array_equal(img.view(np.uint32), ref.view(np.uint32))
