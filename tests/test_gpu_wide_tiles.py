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


@pytest.mark.parametrize("analyser", [False, True])
def test_wide_tiles_take_the_factor_table_by_its_rule(cuda, monkeypatch, analyser):
    """An exposure's wide tiles beyond the factor table's bound take the factor
    per tile; under a top-hat analyser, whose mask is in the table, the sum is
    not the node form's to take."""
    w, sample = _dilute()
    B, st, D = w.beam, StaticStage(w.stage.rotation, w.stage.translation), _det(w, (200, 180))
    plans, runs = [], []
    make, split = engine.NodePlan.make.__func__, engine.run_split
    monkeypatch.setattr(engine.NodePlan, "make", classmethod(
        lambda cls, *a, **k: plans.append(make(cls, *a, **k)) or plans[-1]))
    monkeypatch.setattr(engine, "run_split", lambda *a, **k: runs.append((a, k)) or split(*a, **k))
    kw = dict(apply_polarization=True, return_double=True)
    if analyser:
        kw.update(analyser_mode="top-hat", analyser_acceptance_angle_rad=0.05)
    got = B.atomic_scattering_kinematic(sample, D, st, **kw)
    wide, (tiles, pix, phys, *_), opts = plans[-1].wide, *runs[-1]
    assert wide is not None and not engine.factor_table_ok(wide, pix, phys)
    assert (B.last_run["launch_source"] == "nodes") == (not analyser)
    assert (tiles is wide) == (not analyser) and opts.get("factor_table") is None
    B._use_fast_kernel = False
    ref = B.atomic_scattering_kinematic(sample, D, st, **kw)
    assert rel_intensity(got, ref) <= 1e-4, rel_intensity(got, ref)
