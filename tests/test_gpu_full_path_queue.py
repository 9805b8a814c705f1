"""The full path's queue holds each output sample once: exactly those that fetch at 2R
by the statistics run, and of the ones that outgrew the first light tier perhaps some
that start over.  (A second entry of an output sample changes no colour.)"""
import pytest

import tlfr
from test_gpu_light_scan import CASES, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,opt", CASES, ids=[str(i) for i in range(len(CASES))])
def test_queue_holds_the_2r_fetches_once(kind, opt):
    rec, coc = _scene(kind)
    p = tlfr.CameraParams(overrideUVT=opt.get("uvt"), outputSpp=opt.get("output_spp", 0))
    g = tlfr.TreeGather(tlfr.UVTSampleBuffer(records=rec, coc=coc), p, opt.get("aperture", 1.0), opt.get("focus", 1.0))
    g.reconstructDofMotion()
    timed = g.stats()
    _, counted = g.reconstructDofMotion(stats=True)
    more = timed.num_heavy_queries - counted.num_2r
    assert 0 <= more <= timed.num_retried_queries
    print(f"{int(counted.num_2r)} fetches at 2R, {int(more)} more, {int(timed.num_retried_queries)} retried")
