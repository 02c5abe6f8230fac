"""The adjoint's backward pass where the device memory does not hold a path
slot for every sample: it goes on with fewer (an allocation that fails is
injected on the host), computes the same gradients, and keeps to that size."""
import numpy as np
import pytest

import dort_b200 as db
from dort_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _injection_off():
    yield
    db.debug_fail_alloc(-1)


@pytest.mark.parametrize("point", ["queues", "term log"])
def test_backward_with_fewer_slots(cuda, point):
    sd = scenes.adjoint_scene(n_tris=2000)
    p = db.render_params(sd["camera"], 48, 40, 8, max_depth=3, seed=2)
    alb, em = sd["tri_albedo"], sd["tri_emission"]
    sc = db.scene_from_dict(sd)
    img = sc.adjoint_forward(p, alb, em)
    _, g = db.loss_l2(img, np.zeros_like(img))
    ref_sc = db.scene_from_dict(sd)
    want = ref_sc.adjoint_backward(p, g, alb, em)
    waves = ref_sc.adjoint_stats()["waves"]
    # the gradient buffers come first, then the queues, then the log
    db.debug_fail_alloc({"queues": 1, "term log": 2}[point])
    for _ in range(2):
        got = sc.adjoint_backward(p, g, alb, em)
        db.debug_fail_alloc(-1)
        # 15,360 samples in half as many slots
        assert sc.adjoint_stats()["waves"] > waves
        for a, b in zip(got, want):
            # float atomics add in any order: equal to rounding, in norm
            assert np.abs(b).sum() > 0
            assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b)
