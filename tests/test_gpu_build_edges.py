"""The hierarchy build at the edges of its kernels' cases, node for node against the
oracle: cells of 15 to 200 candidates (sorted in shared memory up to 64, in place
beyond; FW::sort turns from insertion sort to quicksort at 16), samples reprojected to
the shutter's start, middle and end, equal keys, samples with invalid bounds, and grids
with fewer than five kd levels."""
import numpy as np
import pytest

import tlfr
from tlfr_testutil import CpuRecon, compare_trees

pytestmark = pytest.mark.gpu


def _spot(n, seed):
    """n samples within a hundredth of a pixel, with few distinct depths and all three times."""
    rng = np.random.default_rng(seed)
    rec = np.zeros((1, n, 1, 16), np.float32)
    rec[..., 0] = 0.5 + 0.01 * rng.random(rec.shape[:3])
    rec[..., 1] = 0.5 + 0.01 * rng.random(rec.shape[:3])
    w = rng.choice(np.float32([1, 1.5, 2]), rec.shape[:3])
    rec[..., 2] = w
    rec[..., 3] = w
    when = rng.integers(0, 3, rec.shape[:3])
    rec[..., 6] = np.choose(when, [0.0, 0.4, 1.0])
    rec[..., 13] = np.choose(when, [-4.0, 0.0, 4.0]) * w      # w <= 0 at the middle of the shutter
    rec[..., 7:10] = rng.random(rec.shape[:3] + (3,))
    rec[..., 10] = 1
    return rec, (-2.0, 1.5)


def _moving(width, height, spp):
    """Cards with motion fast enough to leave the screen for the whole shutter."""
    rec, coc = tlfr.synth_scene(tlfr.SCENE_CARDS_LARGE, width, height, spp, 9)
    rec[..., 11] *= 8
    rec[..., 12] *= -6
    return rec, coc


CASES = [("spot", n) for n in (3, 15, 16, 17, 48, 49, 63, 64, 65, 200)] + [
    ("moving", (20, 16, 4)), ("moving", (97, 33, 2)), ("moving", (64, 64, 16))]


@pytest.mark.parametrize("kind,size", CASES)
def test_build_edges_match_oracle(kind, size):
    rec, coc = _spot(size, 11) if kind == "spot" else _moving(*size)
    g = tlfr.TreeGather(tlfr.UVTSampleBuffer(records=rec, coc=coc))
    o = CpuRecon("orc", rec, coc)
    for _ in range(2):
        assert compare_trees(g.tree_export(), o.tree()) == []
        g.rebuild_from(tlfr.UVTSampleBuffer(records=rec, coc=coc))
