"""The node form's plan takes the SM count of the device it is for, and its
launches take it from the plan."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import engine, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sms", [1, 13, 1000])
def test_plan_carries_the_sm_count(cuda, sms):
    w = workloads.fcc_cu_32k(cells=20, npix=128)
    B = w.beam
    phys = B.physics(**w.sc_kwargs)
    atoms = B.stage_atoms(w.sample, w.stage, device=cuda)
    pix = engine.Pixels(np.asarray(w.detector.pixel_coordinates) / 1e10, 128, 128, phys, device=cuda)
    tiles = engine.Tiles(atoms, B.k, 512, device=cuda)
    plan = engine.NodePlan.make(tiles, pix, B.k, (1.0, 0.0, 0.0), 1e-6, direct=1.0, group_tiles=8)
    assert plan.plan.sms == torch.cuda.get_device_properties(cuda).multi_processor_count
    want = engine.run_nodes(plan, tiles, pix, phys, atoms.table)
    plan.plan.sms = sms                     # another split of the leaves' patches, the same sums
    got = engine.run_nodes(plan, tiles, pix, phys, atoms.table)
    engine.sync()
    assert torch.equal(got, want)
