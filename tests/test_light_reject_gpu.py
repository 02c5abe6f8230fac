"""The wavefront does not trace BSDF-strategy rays that pass their light's
triangle by; the whole-path kernel traces every one.  The same image and the same
count of rays, also where a light's own triangle differs from the primitive that
emits, with every light sampled, and with the watertight triangle test.  The two
are compiled apart, so a rare path may take another branch: at most two pixels,
and one ray in a thousand, as in the other comparisons of the two."""
import numpy as np
import pytest

import dort_b200 as db
from dort_b200 import scenes

pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("own", [False, True])
@pytest.mark.parametrize("form", ["one", "all", "watertight"])
def test_passed_lights(own, form):
    sd = scenes.cornell_variant("diff", "both")
    emits = np.flatnonzero(np.asarray(sd["tri_emission"]).reshape(-1, 3).any(axis=1))
    assert len(emits)
    if own:
        verts = np.asarray(sd["verts"], np.float32).reshape(-1, 3)
        lv = verts[np.asarray(sd["tris"]).reshape(-1, 3)].copy()
        mid = lv[emits].mean(axis=1, keepdims=True)
        lv[emits] = mid + (lv[emits] - mid) * np.float32(0.5)
        sd["tri_light_verts"] = lv.reshape(-1, 9)
    if form == "watertight":
        sd["watertight"] = True
    sc = db.scene_from_dict(sd)
    p = db.render_params(sd["camera"], 90, 70, 16, max_depth=6, seed=3,
                         sample_all_lights=form == "all")
    mega, st = sc.render(p)
    wave, ws = sc.render_wavefront(p)
    off = np.abs(mega.astype(np.float64) - wave).max(axis=-1) > 1e-4 * mega.mean()
    assert off.sum() <= 2
    assert abs(int(st["rays"]) - int(ws["rays"])) <= 0.001 * st["rays"]
