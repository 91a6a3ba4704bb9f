"""Sums the node form declines build their tiles once, and search no plan
where the detector or the analyser rules it out beforehand."""
import numpy as np
import pytest

from mosaic_gb300 import ChunkedSample, Detector, StaticStage, engine, workloads

from helpers import rel_intensity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("why", ["curved", "direct", "edge"])
def test_a_declined_sum_builds_its_tiles_once(cuda, monkeypatch, why):
    w = workloads.fcc_cu_32k(cells=16, npix=16)
    pos = w.sample.load_chunk_positions(1)
    sample = ChunkedSample([(pos, np.full(len(pos), "Cu"))])
    B = workloads._beam(10000.0, 200.0, pol_perp_rate=1.0)
    st = StaticStage(w.stage.rotation, w.stage.translation)
    D = Detector()
    # 2 mm pixels: a shell is 8 mm off its chord plane at the corners
    pitch = 2.0e7 if why == "curved" else 5.5e5
    D.create_detector((130, 90), (pitch, pitch), construction_mode="shell" if why == "curved" else "plane")
    D.position_detector_absolute(1.0e10, 2.0 * w.meta["theta_deg"], 0.0)
    made, plans = [], []
    tiles, make = engine.Tiles, engine.NodePlan.make.__func__
    monkeypatch.setattr(engine, "Tiles", lambda *a, **k: made.append(tiles(*a, **k)) or made[-1])

    def plan(cls, *a, **k):
        plans.append(make(cls, *a, **dict(k, direct=1e-30 if why == "direct" else 1.0)))
        return plans[-1]
    monkeypatch.setattr(engine.NodePlan, "make", classmethod(plan))
    kw = dict(apply_polarization=True, return_double=True)
    if why == "edge":
        kw.update(analyser_mode="top-hat", analyser_acceptance_angle_rad=3e-3)
        # an edge through a pixel: more edge pixels than are taken
        monkeypatch.setattr(engine, "analyser_mask", lambda *a, **k: None)
    got = B.atomic_scattering_kinematic(sample, D, st, **kw)
    assert B.last_run["launch_source"] != "nodes"
    assert len(made) == 1 and plans == ([None] if why == "direct" else [])
    B._use_fast_kernel = False
    assert rel_intensity(got, B.atomic_scattering_kinematic(sample, D, st, **kw)) <= 1e-4
