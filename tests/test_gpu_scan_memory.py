"""A scan whose node fields do not fit the device runs by the split kernel, as it
would without the node form. The failure is raised by the test at the
allocation."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import engine, workloads
from mosaic_gb300.scan import BatchedScan, frames_from_motors

pytestmark = pytest.mark.gpu


def test_scan_without_room_for_node_fields(cuda, monkeypatch):
    w = workloads.fcc_cu_32k(cells=20, npix=128)
    th = np.radians(w.meta["theta_deg"])
    frames = frames_from_motors(w.stage, w.detector, [dict(mu=th + 1e-3 * i) for i in range(3)], [64, 48, 64])
    direct = BatchedScan(w.beam, w.sample, frames, nodes=False, **w.sc_kwargs)
    sizes, make, empty = [], engine.NodePlan.make.__func__, torch.empty

    def plan(cls, *a, **k):
        p = make(cls, *a, **k)
        sizes.append(p.plan.ws_bytes)
        return p

    def alloc(*a, **k):
        if sizes and a == (sizes[-1],):
            raise torch.cuda.OutOfMemoryError("test")
        return empty(*a, **k)
    monkeypatch.setattr(engine.NodePlan, "make", classmethod(plan))
    monkeypatch.setattr(torch, "empty", alloc)
    scan = BatchedScan(w.beam, w.sample, frames, **w.sc_kwargs)
    monkeypatch.undo()
    assert sizes and scan.nodes is None and scan.launch_source == direct.launch_source
    a, b = scan.run()[0], direct.run()[0]
    engine.sync()
    assert torch.equal(a, b)
