"""The whole-path kernel with few and with several samples per thread (from
four on, a thread starts its next sample while its warp's other paths go on):
the same image as the wavefront, which draws the same random numbers.  The two
are compiled apart, so a rare path may take another branch (at most two pixels,
as in the other comparisons of the two)."""
import numpy as np
import pytest

import dort_b200 as db
from dort_b200 import scenes

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["diff", "glos"])
@pytest.mark.parametrize("per", [1, 3, 4, 5])
def test_samples_per_thread(kind, per):
    w, h = 250, 130
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    slices = sms * 4096 // (w * h)          # the launch plan's slices per pixel
    spp = slices * per - (per > 1)          # the last slice one sample short
    sd = scenes.cornell_variant(kind, "both")
    sc = db.scene_from_dict(sd)
    p = db.render_params(sd["camera"], w, h, spp, max_depth=6, seed=per)
    mega, st = sc.render(p)
    wave, _ = sc.render_wavefront(p)
    assert st["samples"] == w * h * spp
    assert st["dropped"] == 0
    off = np.abs(mega.astype(np.float64) - wave).max(axis=-1) > 1e-4 * mega.mean()
    assert off.sum() <= 2
