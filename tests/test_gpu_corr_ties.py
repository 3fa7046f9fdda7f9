"""Surfaces whose candidates tie along lines or everywhere, bit for bit against
the CPU oracle: whole CTAs of pixels then evaluate chunks of their windows
again, from lists that hold one chunk or all of a pixel's."""
import numpy as np
import pytest

from cudafusion_b200 import synth
from cudafusion_b200.corr import CorrespondenceSearch, CorrParams, DeviceCorrFrame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,radius,chunks,angle", [(160, 96, 20, 1, 0.0), (160, 96, 20, 8, 0.0), (161, 95, 33, 3, 0.3),
                                                     (40, 120, 12, 2, 0.0)])
def test_noise_free_cylinders(oracle, w, h, radius, chunks, angle):
    f = synth.corr_frame(w, h, noise=0.0, seed=radius)
    s = CorrespondenceSearch(w, h)
    s.set_chunks(chunks)
    prm = CorrParams(0.2, angle, 0.0, radius)
    n = s.find_correspondences(DeviceCorrFrame(f), prm, debug=True)
    recs, st = s.records(w * h), s.stats.cpu().numpy()
    ref, nv, rst = oracle.find_correspondences(f, 0.2, angle, 0.0, radius)
    assert n == nv and np.array_equal(st, rst)
    assert np.array_equal(np.ascontiguousarray(recs).view(np.uint8), np.ascontiguousarray(ref).view(np.uint8))
