"""The node form's error at the size it has, not only within the FP32 forms'
gate: against the FP64 sum of the same atoms and pixels.

Tolerances. Two to five factors exp(i phase) a term, each 7.3e-8 short by
__sincosf and corrected to ~1e-8; interpolation at most 3e-8 an axis and step
(1.8e-7 for three steps, of either sign); weights that sum to 1 and a factor
rounded once (6e-8, another at every pixel): the field's scale -- its projection
on the FP64 field -- is within 2e-7 of 1, where the uncorrected factors alone
take 2 to 4e-7. Single pixels add the FP32 phases' rounding (1e-7 cycles a step,
averaged over the atoms): 2e-6 of the peak intensity, and 3e-6 of max |A| against
the split kernel with one sin/cos a term, whose phases are rounded alike. (The
FP64 sum's complex field is no measure of that: it rounds k |P| as the reference
does, k ulp(|P|) = 1.1e-5 rad at 1 m.)"""
import numpy as np
import pytest
import torch

from mosaic_gb300 import ChunkedSample, Detector, StaticStage, engine, workloads

from helpers import rel_intensity, rel_max

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells, shape, dist, tile, group", [
    (14, (64, 48), 1.0e10, 512, 0),         # tiles straight to the pixels
    (24, (128, 96), 1.0e10, 512, 8),        # eighths, groups
    (24, (301, 187), 0.5e10, 512, 8),
    (28, (256, 256), 0.5e10, 256, -1),      # as the plan chooses
    (40, (200, 160), 1.0e10, 512, -1),
])
def test_scale_and_largest_error(cuda, cells, shape, dist, tile, group):
    w = workloads.fcc_cu_32k(cells=cells, npix=16)
    pos = w.sample.load_chunk_positions(1)
    spc = np.where(np.random.default_rng(5).random(len(pos)) < 0.3, "Ni", "Cu")
    B = workloads._beam(10000.0, 200.0, pol_perp_rate=1.0)
    st = StaticStage(w.stage.rotation, w.stage.translation)
    D = Detector()
    D.create_detector(shape, (5.5e5, 5.5e5))
    D.position_detector_absolute(dist, 2.0 * w.meta["theta_deg"], 0.0)
    phys = B.physics(apply_polarization=True)
    atoms = B.stage_atoms(ChunkedSample([(pos, spc)]), st, device=cuda)
    pix = engine.Pixels(np.asarray(D.pixel_coordinates) / 1e10, *shape, phys, device=cuda)
    tiles = engine.Tiles(atoms, B.k, tile, device=cuda)
    plan = engine.NodePlan.make(tiles, pix, B.k, (1.0, 0.0, 0.0), 1e-6, direct=1.0, group_tiles=group)
    assert plan is not None and plan.wide is None
    fresnel = B.split_budget(tiles, pix.r0_min())
    got = engine.run_nodes(plan, tiles, pix, phys, atoms.table, fresnel=int(fresnel[1]),
                           fresnel_radius=fresnel[3]["fresnel_radius_m"])
    ref = engine.run_plain(atoms, pix, phys)
    one = engine.run_split(tiles, pix, phys, atoms.table, fresnel=1)
    engine.sync()
    got, ref, one = (torch.view_as_complex(x).cpu().numpy() for x in (got, ref, one))
    scale = float((got * ref.conj()).sum().real / (np.abs(ref) ** 2).sum()) - 1.0
    print(plan.info(), "scale", scale, "intensity", rel_intensity(got, ref), "field", rel_max(got, one))
    assert abs(scale) <= 2e-7, scale
    assert rel_intensity(got, ref) <= 2e-6
    assert rel_max(got, one) <= 3e-6
