"""An edited frame's pixels are the ones a batched scan takes; the other frames
of its ROI keep theirs."""
import numpy as np
import pytest

from mosaic_gb300 import workloads
from mosaic_gb300.scan import BatchedScan, frames_from_motors

pytestmark = pytest.mark.gpu


def test_scan_takes_edited_pixels(cuda):
    w = workloads.fcc_cu_32k(cells=6, npix=32)
    th = np.radians(w.meta["theta_deg"])
    frames = frames_from_motors(w.stage, w.detector, [dict(mu=th)] * 3, [8, 8, 8])
    frames[1].pixels[2] += 1.0e6            # 0.1 mm
    xyz = BatchedScan(w.beam, w.sample, frames, **w.sc_kwargs).pix.xyz.cpu().numpy().reshape(3, 64, 3)
    R = np.asarray(frames[0].rotation, np.float64)
    assert np.array_equal(xyz[0], xyz[2])
    assert np.allclose((xyz[1] - xyz[0]) @ R.T, [0.0, 0.0, 1.0e-4], atol=1e-12)
