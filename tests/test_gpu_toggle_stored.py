"""The GPU-toggle algorithm against stored images, where the reference build is absent:
tests/golden/toggle/images.npz holds this library's images of these scenes from a build
that agreed with the reference's own CPU restatement (tests/test_gpu_toggle.py).  Bit
for bit.  One scene crowds single-sample surfaces, so that 2R searches at its edge
outgrow the per-thread leaf lists."""
import os

import numpy as np
import pytest

import tlfr
from tlfr_testutil import GOLDEN

IMAGES = os.path.join(GOLDEN, "toggle", "images.npz")

SCENES = {
    "cards": (tlfr.SCENE_CARDS, 24, 18, 4, 81, {}),
    "large": (tlfr.SCENE_CARDS_LARGE, 28, 20, 8, 82, {}),
    "planes": (tlfr.SCENE_PLANES, 20, 16, 16, 83, {}),
    "one_sample": (tlfr.SCENE_CARDS, 26, 18, 1, 84, {}),
    "refocus": (tlfr.SCENE_CARDS_LARGE, 26, 18, 2, 85, dict(aperture=1.5, focus=0.8)),
    "pinhole": (tlfr.SCENE_CARDS, 32, 24, 4, 86, dict(uvt=(0.0, 0.0, 1.0))),
    "dense": (tlfr.SCENE_CARDS, 20, 16, 8, 87, dict(uvt=(0.0, 0.0, 1.0), scale=0.27)),
}


def render(name):
    """(image, output samples that outgrew the per-thread lists)"""
    preset, w, h, spp, seed, o = SCENES[name]
    rec, coc = tlfr.synth_scene(preset, w, h, spp, seed)
    if "scale" in o:
        # static samples at random depths (a surface each), drawn together
        z = np.exp(np.random.default_rng(seed).uniform(-4, 6, rec.shape[:3])).astype(np.float32)
        rec[..., 2:4] = z[..., None]
        rec[..., 4:6] = 0.0
        rec[..., 11:14] = 0.0
        centre = np.float32([w / 2, h / 2])
        rec[..., :2] = centre + np.float32(o["scale"]) * (rec[..., :2] - centre)
    p = tlfr.CameraParams(enableCuda=True, overrideUVT=o.get("uvt"))
    g = tlfr.TreeGather(tlfr.UVTSampleBuffer(records=rec, coc=coc), p, o.get("aperture", 1.0), o.get("focus", 1.0))
    return g.reconstructDofMotion(), g.stats().num_overflow_queries


@pytest.mark.gpu
@pytest.mark.parametrize("name", SCENES)
def test_gpu_toggle_matches_stored_image(name):
    img, outgrown = render(name)
    assert np.array_equal(img.view(np.uint32), np.load(IMAGES)[name].view(np.uint32))
    assert (outgrown > 0) == (name == "dense")
