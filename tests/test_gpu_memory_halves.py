"""Sums that run out of device memory twice: scatter_device sums the atoms in
halves, and halves of those, into one field, so a sum that fails must not have
added anything yet.

The failures are raised by the test at the allocations. Tolerance: 2e-5 of max
|A| between the FP32 sums of the same atoms whole and in parts (a sum added
twice is off by the order of 1)."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import ChunkedSample, Detector, StaticStage, engine, workloads

from helpers import rel_max

pytestmark = pytest.mark.gpu


def _setup(cells, dist, shape):
    w = workloads.fcc_cu_32k(cells=cells, npix=16)
    pos = w.sample.load_chunk_positions(1)
    spc = np.full(pos.shape[0], "Cu")
    spc[::200] = "Ag"
    D = Detector()
    D.create_detector(shape, (5.5e5, 5.5e5))
    D.position_detector_absolute(dist, 2.0 * w.meta["theta_deg"], 0.0)
    B = workloads._beam(10000.0, 200.0, pol_perp_rate=1.0)
    return B, ChunkedSample([(pos, spc)]), D, StaticStage(w.stage.rotation, w.stage.translation)


def _always_nodes(monkeypatch):
    """Every sum planned in node form; the plans made."""
    plans, make = [], engine.NodePlan.make.__func__

    def forced(cls, *a, **kw):
        plans.append(make(cls, *a, **dict(kw, direct=1.0)))
        return plans[-1]
    monkeypatch.setattr(engine.NodePlan, "make", classmethod(forced))
    return plans


def test_wide_tiles_are_added_once(cuda, monkeypatch):
    B, sample, D, st = _setup(32, 0.05e10, (96, 96))
    kw = dict(apply_polarization=True, return_double=True)
    plans = _always_nodes(monkeypatch)
    whole = B.atomic_scattering_kinematic(sample, D, st, **kw)
    assert B.last_run["launch_source"] == "nodes"
    del plans[:]
    empty, failed = torch.empty, []

    def failing(*a, **k):
        if len(failed) < 2 and plans and a == (plans[-1].plan.ws_bytes,):
            failed.append(plans[-1].wide is not None)
            raise torch.cuda.OutOfMemoryError("test")
        return empty(*a, **k)
    monkeypatch.setattr(torch, "empty", failing)
    parts = B.atomic_scattering_kinematic(sample, D, st, **kw)
    assert failed == [True, True]           # whole, then the first half, both with wide tiles
    assert B.last_run["memory_splits"] >= 1
    assert rel_max(parts, whole) <= 2e-5, rel_max(parts, whole)


def test_top_hat_edge_pixels_are_added_once(cuda, monkeypatch):
    shape = (120, 90)
    B, sample, D, st = _setup(24, 1.0e10, shape)
    xyz = np.asarray(D.pixel_coordinates, np.float64) / 1e10
    c = (np.asarray(D.pixel_coordinates)[:, 45 * 120 + 60].astype(np.float32) / np.float32(1e10)).astype(np.float64)
    c /= np.linalg.norm(c)
    u = xyz[:, 30 * 120 + 17] / np.linalg.norm(xyz[:, 30 * 120 + 17])
    kw = dict(apply_polarization=True, return_double=True, analyser_mode="top-hat",
              analyser_acceptance_angle_rad=2.0 * np.arcsin(0.5 * np.linalg.norm(u - c)))
    _always_nodes(monkeypatch)
    whole = B.atomic_scattering_kinematic(sample, D, st, **kw)
    assert B.last_run["launch_source"] == "nodes" and B.last_run["edge_pixels"] >= 1
    split, plain, failed = engine.run_split, engine.run_plain, []

    def failing(run):           # the edge pixels' sum, whichever kernel it takes
        def call(*a, **k):
            if len(failed) < 2:
                failed.append(1)
                raise torch.cuda.OutOfMemoryError("test")
            return run(*a, **k)
        return call
    monkeypatch.setattr(engine, "run_split", failing(split))
    monkeypatch.setattr(engine, "run_plain", failing(plain))
    parts = B.atomic_scattering_kinematic(sample, D, st, **kw)
    assert len(failed) == 2 and B.last_run["memory_splits"] >= 1
    assert rel_max(parts, whole) <= 2e-5, rel_max(parts, whole)
