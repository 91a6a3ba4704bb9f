"""Sums in node form whose widest tiles -- a dilute species' -- go to the split
kernel, at distances where the groups' directions stay within the factor
table's bound and the wide tiles' do not.

Tolerance: 1e-4 of the peak intensity against FP64, the FP32 forms'."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import ChunkedSample, Detector, StaticStage, engine, workloads
from mosaic_gb300.scan import BatchedScan, frames_from_motors

from helpers import rel_intensity

pytestmark = pytest.mark.gpu

DIST = 0.042e10         # 14.5 nm of crystal: the groups' directions below 1e-6, the widest tiles' above


def _dilute():
    """256,000 fcc sites, 1,024 of them (two tiles) of another species."""
    w = workloads.fcc_cu_32k(cells=40, npix=16)
    pos = w.sample.load_chunk_positions(1)
    spc = np.full(pos.shape[0], "Cu")
    spc[np.random.default_rng(1).choice(pos.shape[0], 1024, replace=False)] = "Ag"
    return w, ChunkedSample([(pos, spc)])


def _det(w, shape):
    D = Detector()
    D.create_detector(shape, (5.5e5, 5.5e5))
    D.position_detector_absolute(DIST, 2.0 * w.meta["theta_deg"], 0.0)
    return D


def test_scan_with_wide_tiles_takes_every_frames_own_factors(cuda):
    w, sample = _dilute()
    B = w.beam
    theta = np.radians(w.meta["theta_deg"])
    steps = [dict(mu=theta + np.radians(0.1 * i - 0.4), chi=np.radians(0.1 * i)) for i in range(8)]
    frames = frames_from_motors(w.stage, _det(w, (128, 128)), steps, [128, 48] + [128] * 6)
    scan = BatchedScan(B, sample, frames, apply_polarization=True)
    assert scan.nodes is not None and scan.nodes.wide is not None
    assert not engine.factor_table_ok(scan.nodes.wide, scan.pix, scan.phys)     # split: factor per tile
    scan.run()
    engine.sync()
    B._use_fast_kernel = False
    for f in (1, 7):
        fr = frames[f]
        ref = B.interact_beam_gpu(sample, fr.pixels, fr.shape, StaticStage(fr.rotation, fr.translation),
                                  apply_polarization=True, spherical_decay=False, return_double=True)
        assert rel_intensity(scan.frame_field(f), ref) <= 1e-4, (f, rel_intensity(scan.frame_field(f), ref))
    # a rotated frame's pixels have no single factor table to fall back on
    with pytest.raises(ValueError):
        engine.run_nodes(scan.nodes, scan.tiles, scan.pix, scan.phys, scan.table)
