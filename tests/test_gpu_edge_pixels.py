"""Pixels that a top-hat analyser's edge cuts, beside the node form: by the split
kernel's per-atom test, against the FP64 sum of every (atom, pixel).

Tolerance: 1e-4 of the peak intensity without the analyser, the FP32 forms'."""
import numpy as np
import pytest

from mosaic_gb300 import ChunkedSample, Detector, StaticStage, engine, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells, shape, dist", [
    (20, (128, 128), 1.0e10),
    (28, (121, 90), 0.5e10),
    (40, (64, 64), 0.2e10),         # a wide edge: many pixels
])
def test_edge_pixels_by_the_split_kernel(cuda, monkeypatch, cells, shape, dist):
    w = workloads.fcc_cu_32k(cells=cells, npix=16)
    pos = w.sample.load_chunk_positions(1)
    sample = ChunkedSample([(pos, np.where(np.arange(len(pos)) % 7 == 0, "Ni", "Cu"))])
    B = workloads._beam(10000.0, 200.0, pol_perp_rate=1.0)
    st = StaticStage(w.stage.rotation, w.stage.translation)
    D = Detector()
    D.create_detector(shape, (5.5e5, 5.5e5))
    D.position_detector_absolute(dist, 2.0 * w.meta["theta_deg"], 0.0)
    ny, nz = shape
    px = np.asarray(D.pixel_coordinates)
    xyz = px.astype(np.float64) / 1e10
    c = (px[:, (nz // 2) * ny + ny // 2].astype(np.float32) / np.float32(1e10)).astype(np.float64)
    c /= np.linalg.norm(c)
    i = (nz // 3) * ny + ny // 7
    u = xyz[:, i] / np.linalg.norm(xyz[:, i])
    kw = dict(apply_polarization=True, spherical_decay=True, return_double=True)
    ana = dict(kw, analyser_mode="top-hat",
               analyser_acceptance_angle_rad=2.0 * np.arcsin(0.5 * np.linalg.norm(u - c)))
    plain = []
    run = engine.run_plain
    monkeypatch.setattr(engine, "run_plain", lambda *a, **k: plain.append(1) or run(*a, **k))
    got = B.atomic_scattering_kinematic(sample, D, st, **ana)
    assert B.last_run["launch_source"] == "nodes" and B.last_run["edge_pixels"] >= 1, B.last_run
    assert not plain                        # a pixel costs the FP64 sum a warp's time for every atom
    again = B.atomic_scattering_kinematic(sample, D, st, **ana)
    assert np.array_equal(got, again)
    B._use_fast_kernel = False
    ref = B.atomic_scattering_kinematic(sample, D, st, **ana)
    peak = (np.abs(B.atomic_scattering_kinematic(sample, D, st, **kw)) ** 2).max()
    assert np.abs(np.abs(got) ** 2 - np.abs(ref) ** 2).max() <= 1e-4 * peak
    assert ((got == 0) == (ref == 0)).all()
