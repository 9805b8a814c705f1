"""Samples at the ends of single precision's range of depths, against the oracle bit
for bit: w around and beyond 2^126, where the hardware's approximate reciprocal has no
normal result, beside samples of the scene's own depths."""
import numpy as np
import pytest

import tlfr
from tlfr_testutil import CpuRecon

pytestmark = pytest.mark.gpu

# (w, corner): x, y < corner keep x * w finite
FAR = [(1e30, 12), (8.0e37, 4), (8.5e37, 4), (8.6e37, 3), (1e38, 3), (3.4e38, 1)]


@pytest.mark.parametrize("uvt", [None, (0.0, 0.0, 1.0)], ids=["lens", "pinhole"])
@pytest.mark.parametrize("w,corner", FAR)
def test_far_samples_match_oracle(w, corner, uvt):
    rec, coc = tlfr.synth_scene(tlfr.SCENE_CARDS, 12, 10, 8, 3)
    far = rec[:corner, :corner, ::2]
    far[..., 2:4] = w
    far[..., 4:6] = 0.0
    far[..., 11:14] = 0.0
    coc = (coc[0], 0.1 * coc[1])
    g = tlfr.TreeGather(tlfr.UVTSampleBuffer(records=rec, coc=coc), tlfr.CameraParams(overrideUVT=uvt))
    ref = CpuRecon("orc", rec, coc, uvt=uvt).reconstruct()
    assert np.array_equal(g.reconstructDofMotion().view(np.uint32), ref.view(np.uint32))
