"""The light pass's scan at its edges, against the oracle bit for bit: more samples
set aside per output sample than its list holds, leaves of hundreds of samples,
equal sort keys, output samples outside the lens and the shutter (where the
approximate radius test has the widest bounds), and circles of confusion large
against the image."""
import numpy as np
import pytest

import tlfr
from tlfr_testutil import CpuRecon

pytestmark = pytest.mark.gpu


def _scene(kind):
    if kind == "one_spot":
        # every sample within a hundredth of a pixel: one grid cell, leaves of hundreds of samples
        rec, coc = tlfr.synth_scene(tlfr.SCENE_CARDS, 12, 10, 16, 5)
        rng = np.random.default_rng(1)
        rec[..., 0] = 5.5 + 0.01 * rng.random(rec.shape[:3], dtype=np.float32)
        rec[..., 1] = 4.5 + 0.01 * rng.random(rec.shape[:3], dtype=np.float32)
        rec[..., 2:4] = 3.0
        rec[..., 4:6] = 0.0
        rec[..., 11:14] = 0.0
        return rec, coc
    if kind == "flat":
        # one static plane: every leaf's key is the same
        rec, coc = tlfr.synth_scene(tlfr.SCENE_CARDS, 40, 24, 8, 6)
        rec[..., 2:4] = 2.5
        rec[..., 11:14] = 0.0
        return rec, coc
    preset, w, h, s = kind
    return tlfr.synth_scene(preset, w, h, s, 7)


CASES = [
    ("one_spot", {}),
    ("one_spot", dict(aperture=0.1)),
    ("flat", {}),
    ((tlfr.SCENE_CARDS, 16, 12, 3), {}),
    ((tlfr.SCENE_CARDS, 14, 11, 12), {}),       # dispersion 2 at 12 samples per pixel: about 150 within the radius
    ((tlfr.SCENE_PLANES, 17, 13, 24), dict(output_spp=20)),
    ((tlfr.SCENE_CARDS_LARGE, 33, 9, 8), dict(aperture=3.0, focus=0.4)),
    ((tlfr.SCENE_CARDS_LARGE, 31, 19, 8), dict(uvt=(1.1, -1.05, 1.0))),
    ((tlfr.SCENE_CARDS, 31, 19, 8), dict(uvt=(1.15, -1.2, 1.02))),
    ((tlfr.SCENE_PLANES, 31, 19, 8), dict(uvt=(1.3, -1.2, 2.0))),
    ((tlfr.SCENE_CARDS, 31, 19, 8), dict(uvt=(-0.6, 0.8, -0.02))),
]


@pytest.mark.parametrize("kind,opt", CASES, ids=[str(i) for i in range(len(CASES))])
def test_light_scan_edges_match_oracle(kind, opt):
    rec, coc = _scene(kind)
    p = tlfr.CameraParams(overrideUVT=opt.get("uvt"), outputSpp=opt.get("output_spp", 0))
    g = tlfr.TreeGather(tlfr.UVTSampleBuffer(records=rec, coc=coc), p, opt.get("aperture", 1.0), opt.get("focus", 1.0))
    img = g.reconstructDofMotion()
    ref = CpuRecon("orc", rec, coc, **opt).reconstruct()
    assert np.array_equal(img.view(np.uint32), ref.view(np.uint32))
    # an output sample is queued for the full path once, also when the scan's list
    # fills up inside another one of its warp (the queue holds one entry for each)
    outputs = img.shape[0] * img.shape[1] * (1 if p.overrideUVT else p.outputSpp or 128)
    assert g.stats().num_heavy_queries <= outputs


@pytest.mark.parametrize("seed", [6, 1235])
def test_full_size_frame_equals_the_counting_path(seed):
    """Every pixel of the strong-blur frame at 1920x1080x8: the passes of the timed path
    against the statistics run, which takes every output sample through the reference's
    full algorithm, one thread each.  (Differences of one rounding in a node's planes show
    in a few output samples of a quarter of a billion.)"""
    rec, coc = tlfr.synth_scene(tlfr.SCENE_CARDS_LARGE, 1920, 1080, 8, seed)
    g = tlfr.TreeGather(tlfr.UVTSampleBuffer(records=rec, coc=coc))
    img = g.reconstructDofMotion()
    ref, _ = g.reconstructDofMotion(stats=True)
    assert np.array_equal(img.view(np.uint32), ref.view(np.uint32))
