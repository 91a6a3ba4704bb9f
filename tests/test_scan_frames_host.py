"""Frames of a scan made from motor steps: every ROI frame's pixels are its own
to edit."""
import dataclasses

import numpy as np

from mosaic_gb300 import workloads
from mosaic_gb300.scan import Frame, frames_from_motors


def test_frames_of_one_roi_are_edited_by_themselves():
    w = workloads.fcc_cu_32k(cells=2, npix=32)
    steps = [dict(mu=0.1 * i) for i in range(4)]
    a, b, c, full = frames_from_motors(w.stage, w.detector, steps, [8, 8, 8, None])
    want = np.array(a.source())
    assert want.shape == (3, 64) and full.pixels.shape == (3, 1024)
    assert a.source() is b.source()             # one array until a frame's is read
    b.pixels[0] += 5.0
    assert np.array_equal(a.pixels, want) and np.array_equal(c.pixels, want)
    assert np.array_equal(b.source(), want + np.array([[5.0], [0.0], [0.0]]))
    c.pixels = want[:, ::-1]
    assert np.array_equal(c.source(), want[:, ::-1]) and np.array_equal(a.source(), want)
    d = dataclasses.replace(b, shape=(4, 16))
    assert isinstance(d, Frame) and d.shape == (4, 16) and np.array_equal(d.pixels, b.pixels)
