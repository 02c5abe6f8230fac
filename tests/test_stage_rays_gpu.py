"""The ray counts of a wavefront frame: the total is the paths' (the
megakernel's count), the stages' are the rays they traced.  Under a sky all of
a path's rays are traced; under a triangle light the BSDF-strategy rays that
pass the light by are not."""
import pytest

import dort_b200 as db
from dort_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lit_by", ["sky", "triangles"])
def test_stage_rays_are_the_rays_traced(cuda, lit_by):
    sd = scenes.wavefront_scene(12) if lit_by == "sky" else scenes.cornell_box()
    sc = db.scene_from_dict(sd)
    p = db.render_params(sd["camera"], 96, 64, 4, max_depth=5, seed=9)
    st = sc.wavefront_stage_times(p)
    _, frame = sc.render_wavefront(p)
    assert st["rays"] == frame["rays"]
    traced = st["extend_rays"] + st["shadow_rays"] + st["neeb_rays"]
    assert min(st["extend_rays"], st["shadow_rays"]) > 0
    if lit_by == "sky":
        assert traced == st["rays"]
    else:
        # most of the diffuse walls' BSDF-strategy rays miss a light of 0.25 m2
        assert traced < 0.95 * st["rays"]
