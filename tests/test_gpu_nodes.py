"""The node form of the FP32 sum (engine.NodePlan / run_nodes) against the
FP64 sum of the same atoms and pixels and against the split kernel with one
sin/cos per term.

Tolerances are the other FP32 forms': 1e-4 of the peak intensity against
FP64, 2e-5 of max |A| against the one-sin/cos form (interpolation adds at
most ~1e-6 of the sum of |E| by the plan's node counts)."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import ChunkedSample, Detector, StaticStage, engine, workloads
from mosaic_gb300.scan import BatchedScan, frames_from_motors

from helpers import rel_intensity, rel_max

pytestmark = pytest.mark.gpu


def _case(cells, dilute=0.0, seed=3):
    rng = np.random.default_rng(seed)
    w = workloads.fcc_cu_32k(cells=cells, npix=16)
    pos = w.sample.load_chunk_positions(1)
    u = rng.random(pos.shape[0])
    spc = np.where(u < dilute, "Ag", np.where(u < 0.4, "Ni", "Cu"))
    return w, ChunkedSample([(pos, spc)])


def _det(w, shape, dist=1.0e10, mode="plane", pitch=5.5e5):
    D = Detector()
    D.create_detector(shape, (pitch, pitch), construction_mode=mode)
    D.position_detector_absolute(dist, 2.0 * w.meta["theta_deg"], 0.0)
    return D


def _c(out, shape):
    engine.sync()
    return torch.view_as_complex(out).cpu().numpy().reshape(shape[1], shape[0])


@pytest.mark.parametrize("shape, tile, group, dist, decay, cplx", [
    ((64, 48), 512, 0, 1.0e10, False, False),     # one patch, tiles straight to the pixels
    ((33, 17), 128, 0, 1.0e10, True, True),       # one past a pixel block each way, complex amplitudes
    ((1, 40), 128, 0, 1.0e10, False, False),      # single column
    ((50, 1), 128, 0, 1.0e10, False, False),      # single row
    ((200, 90), 128, 8, 0.2e10, True, False),     # groups, several patches, last ones ragged
    ((96, 64), 128, 16, 0.2e10, False, True),     # whole blocks
    ((161, 47), 256, 8, 0.5e10, True, True),
])
def test_nodes_match_fp64_and_split(cuda, shape, tile, group, dist, decay, cplx):
    w, sample = _case(14, dilute=0.005 if group else 0.0)
    B = workloads._beam(10000.0, 200.0, pol_perp_rate=1.0)
    if cplx:
        rng = np.random.default_rng(2)
        B.set_wavefield((B._beam_E0_map * np.exp(1j * rng.uniform(-np.pi, np.pi, B._beam_E0_map.shape))
                         ).astype(np.complex64))
    B.set_debye_waller({"Cu": 0.55})
    st = StaticStage(w.stage.rotation, w.stage.translation)
    D = _det(w, shape, dist)
    phys = B.physics(apply_polarization=True, spherical_decay=decay)
    atoms = B.stage_atoms(sample, st, device=cuda)
    pix = engine.Pixels(np.asarray(D.pixel_coordinates) / 1e10, *shape, phys, device=cuda)
    tiles = engine.Tiles(atoms, B.k, tile, device=cuda)
    plan = engine.NodePlan.make(tiles, pix, B.k, (1.0, 0.0, 0.0), 1e-6, direct=1.0, group_tiles=group)
    assert plan is not None and (plan.plan.n_groups > 0) == (group > 0)
    assert plan.plan.n_members + plan.plan.n_mid + plan.plan.n_wide == tiles.n_tiles
    acc = torch.full((pix.n, 2), float("nan"), dtype=torch.float64, device=cuda)
    wide = plan.wide is not None
    if wide:
        engine.run_split(plan.wide, pix, phys, atoms.table, fresnel=1, out=acc, factor_table=True)
    got = _c(engine.run_nodes(plan, tiles, pix, phys, atoms.table, out=acc, accumulate=wide, fresnel=1), shape)
    one = _c(engine.run_split(tiles, pix, phys, atoms.table, fresnel=1), shape)
    ref = _c(engine.run_plain(atoms, pix, phys), shape)
    assert rel_intensity(got, ref) <= 1e-4, rel_intensity(got, ref)
    assert rel_max(got, one) <= 2e-5, rel_max(got, one)
    again = engine.run_nodes(plan, tiles, pix, phys, atoms.table, fresnel=1)
    engine.sync()
    if not wide:
        assert torch.equal(again, acc)              # the same sum twice, to the bit


@pytest.mark.parametrize("cells, dilute, shape, dist, n0", [
    (24, 0.005, (200, 90), 0.2e10, 20),     # dilute tiles among the groups: eighths too wide for their nodes
    (20, 0.02, (257, 33), 0.5e10, 16),
    (24, 0.0, (400, 130), 0.1e10, 20),      # several coarse patches, tiles with the |d|^2 term
])
def test_leaf_by_eighths_matches_fp64_and_split(cuda, cells, dilute, shape, dist, n0):
    """Tiles of 512 atoms whose coarse nodes are filled from their eighths'."""
    w, sample = _case(cells, dilute=dilute)
    B = workloads._beam(10000.0, 200.0, pol_perp_rate=1.0)
    st = StaticStage(w.stage.rotation, w.stage.translation)
    D = _det(w, shape, dist)
    phys = B.physics(apply_polarization=True)
    atoms = B.stage_atoms(sample, st, device=cuda)
    pix = engine.Pixels(np.asarray(D.pixel_coordinates) / 1e10, *shape, phys, device=cuda)
    tiles = engine.Tiles(atoms, B.k, 512, device=cuda)
    plan = engine.NodePlan.make(tiles, pix, B.k, (1.0, 0.0, 0.0), 1e-6, direct=1.0, group_tiles=8)
    assert plan is not None and plan.plan.n0 == n0 and plan.plan.ns[0] > 0 and plan.plan.n_members > 0
    acc = torch.full((pix.n, 2), float("nan"), dtype=torch.float64, device=cuda)
    wide = plan.wide is not None
    if wide:
        engine.run_split(plan.wide, pix, phys, atoms.table, fresnel=1, out=acc, factor_table=True)
    got = _c(engine.run_nodes(plan, tiles, pix, phys, atoms.table, out=acc, accumulate=wide, fresnel=1), shape)
    one = _c(engine.run_split(tiles, pix, phys, atoms.table, fresnel=1), shape)
    ref = _c(engine.run_plain(atoms, pix, phys), shape)
    assert rel_intensity(got, ref) <= 1e-4, rel_intensity(got, ref)
    assert rel_max(got, one) <= 2e-5, rel_max(got, one)


@pytest.mark.parametrize("cells, dilute, tile, shape, dist", [
    (28, 0.01, 256, (256, 256), 0.2e10),
    (24, 0.0, 512, (301, 187), 0.2e10),
    (24, 0.0, 128, (256, 256), 0.1e10),     # tiles on the fine nodes and wide ones too
])
def test_middle_level_matches_fp64_and_split(cuda, cells, dilute, tile, shape, dist):
    """Tiles merged into runs on middle nodes, single tiles among them, and
    those into groups."""
    w, sample = _case(cells, dilute=dilute)
    B = workloads._beam(10000.0, 200.0, pol_perp_rate=1.0)
    st = StaticStage(w.stage.rotation, w.stage.translation)
    D = _det(w, shape, dist)
    phys = B.physics(apply_polarization=True)
    atoms = B.stage_atoms(sample, st, device=cuda)
    pix = engine.Pixels(np.asarray(D.pixel_coordinates) / 1e10, *shape, phys, device=cuda)
    tiles = engine.Tiles(atoms, B.k, tile, device=cuda)
    plan = engine.NodePlan.make(tiles, pix, B.k, (1.0, 0.0, 0.0), 1e-6, direct=1.0)
    assert plan is not None and plan.plan.nm > 0 and plan.plan.n_msingle > 0
    acc = torch.full((pix.n, 2), float("nan"), dtype=torch.float64, device=cuda)
    wide = plan.wide is not None
    if wide:
        engine.run_split(plan.wide, pix, phys, atoms.table, fresnel=1, out=acc, factor_table=True)
    got = _c(engine.run_nodes(plan, tiles, pix, phys, atoms.table, out=acc, accumulate=wide, fresnel=1), shape)
    one = _c(engine.run_split(tiles, pix, phys, atoms.table, fresnel=1), shape)
    ref = _c(engine.run_plain(atoms, pix, phys), shape)
    assert rel_intensity(got, ref) <= 1e-4, rel_intensity(got, ref)
    assert rel_max(got, one) <= 2e-5, rel_max(got, one)


def test_entry_point_takes_nodes_where_admitted(cuda):
    """Large enough on a plane detector: nodes; a curved (shell) detector,
    an explicit launch, remove_forward and a Darwin analyser: the other forms,
    with the same field where the physics is the same."""
    w, sample = _case(16)
    B = workloads._beam(10000.0, 200.0, pol_perp_rate=1.0)
    st = StaticStage(w.stage.rotation, w.stage.translation)
    kw = dict(apply_polarization=True, return_double=True)
    D = _det(w, (130, 90))
    a = B.atomic_scattering_kinematic(sample, D, st, **kw)
    assert B.last_run["launch_source"] == "nodes" and B.last_run["path"] == "split_f32"
    B._kernel_launch = dict(pix_per_thread=4, threads=128, slices=0, pairs=0)
    b = B.atomic_scattering_kinematic(sample, D, st, **kw)
    assert B.last_run["launch_source"] == "beam"
    assert rel_max(a, b) <= 2e-5, rel_max(a, b)
    B._kernel_launch = None
    for extra in (dict(remove_forward=True), dict(analyser_mode="darwin", analyser_darwin_halfwidth_rad=1e-3)):
        B.atomic_scattering_kinematic(sample, D, st, **kw, **extra)
        assert B.last_run["launch_source"] != "nodes", extra
    # 2 mm pixels: the sphere is 8 mm off its chord plane at the corners
    S = _det(w, (130, 90), mode="shell", pitch=2.0e7)
    c = B.atomic_scattering_kinematic(sample, S, st, **kw)
    assert B.last_run["launch_source"] != "nodes"
    B._use_fast_kernel = False
    assert rel_intensity(c, B.atomic_scattering_kinematic(sample, S, st, **kw)) <= 1e-4


def test_scan_nodes_match_single_fp64_exposures(cuda):
    """Frames of several shapes in one node plan, their sums, and a captured
    replay, bit for bit."""
    w, sample = _case(16)
    B = w.beam
    theta = np.radians(w.meta["theta_deg"])
    D = _det(w, (128, 128))
    steps = [dict(mu=theta + np.radians(d), chi=np.radians(c)) for c in (-0.3, 0.2) for d in (-0.5, 0.0, 0.4)]
    frames = frames_from_motors(w.stage, D, steps, [24, 128, 50, 64, 33, 128])
    scan = BatchedScan(B, sample, frames, apply_polarization=True)
    assert scan.launch_source == "nodes" and scan.nodes is not None
    out, sums = scan.run()
    engine.sync()
    first, s1 = out.clone(), sums.clone()
    B._use_fast_kernel = False
    for f, fr in enumerate(frames):
        ref = B.interact_beam_gpu(sample, fr.pixels, fr.shape, StaticStage(fr.rotation, fr.translation),
                                  apply_polarization=True, spherical_decay=False, return_double=True)
        assert rel_intensity(scan.frame_field(f), ref) <= 1e-4, f
        I = float((np.abs(scan.frame_field(f)) ** 2).sum())
        assert abs(float(s1[f]) - I) <= 1e-12 * I
    scan.capture()
    scan.out.zero_()
    scan.replay()
    torch.cuda.synchronize()
    assert torch.equal(scan.out, first) and torch.equal(scan.sums, s1)


@pytest.mark.parametrize("npix, dist, n0", [(48, 0.5e10, 8), (32, 0.2e10, 10), (48, 0.2e10, 12), (96, 0.2e10, 16),
                                            (128, 0.2e10, 20)])
def test_eighths_of_either_class_match_the_direct_sum(cuda, npix, dist, n0):
    """Enough tiles and frames for two classes of tiles, on every count of
    coarse nodes: the scan in node form against the scan by the split kernel,
    and one frame against FP64."""
    w, sample = _case(28)
    B = w.beam
    theta = np.radians(w.meta["theta_deg"])
    frames = frames_from_motors(w.stage, _det(w, (128, 128), dist), [dict(mu=theta + np.radians(0.1 * i)) for i in range(12)],
                                [npix] * 12)
    scan = BatchedScan(B, sample, frames, apply_polarization=True)
    plan = scan.nodes.plan
    assert plan.n0 == n0 and plan.ns[0] > 0 and 0 < plan.n_narrow <= plan.n_members
    assert (plan.ns[1] > 0) == (n0 >= 12)
    got = scan.run()[0].clone()
    direct = BatchedScan(B, sample, frames, apply_polarization=True, nodes=False)
    ref = direct.run()[0]
    engine.sync()
    assert float((got - ref).norm(dim=1).max() / ref.norm(dim=1).max()) <= 2e-5
    B._use_fast_kernel = False
    exact = B.interact_beam_gpu(sample, frames[5].pixels, frames[5].shape,
                                StaticStage(frames[5].rotation, frames[5].translation),
                                apply_polarization=True, spherical_decay=False, return_double=True)
    assert rel_intensity(scan.frame_field(5), exact) <= 1e-4


@pytest.mark.parametrize("acceptance", [0.0, 1.1e-3, "edge", 1.0])
def test_top_hat_nodes_match_fp64(cuda, acceptance):
    """A top-hat analyser in the factor table: nothing, some and everything
    accepted, and an edge through one pixel's atoms (that pixel goes to the
    FP64 sum), against the FP64 sum of every (atom, pixel)."""
    w, sample = _case(16)
    B = workloads._beam(10000.0, 200.0, pol_perp_rate=1.0)
    st = StaticStage(w.stage.rotation, w.stage.translation)
    shape = (120, 90)
    D = _det(w, shape)
    xyz = np.asarray(D.pixel_coordinates, np.float64) / 1e10
    c = (np.asarray(D.pixel_coordinates)[:, 45 * 120 + 60].astype(np.float32) / np.float32(1e10)).astype(np.float64)
    c /= np.linalg.norm(c)
    if acceptance == "edge":
        u = xyz[:, 30 * 120 + 17] / np.linalg.norm(xyz[:, 30 * 120 + 17])
        acceptance = 2.0 * np.arcsin(0.5 * np.linalg.norm(u - c))
    kw = dict(apply_polarization=True, spherical_decay=True, return_double=True, analyser_mode="top-hat",
              analyser_acceptance_angle_rad=acceptance)
    got = B.atomic_scattering_kinematic(sample, D, st, **kw)
    run = dict(B.last_run)
    assert run["launch_source"] == "nodes", run
    if acceptance not in (0.0, 1.1e-3, 1.0):
        assert 1 <= run["edge_pixels"] <= 8, run
    B._use_fast_kernel = False
    ref = B.atomic_scattering_kinematic(sample, D, st, **kw)
    one = B.atomic_scattering_kinematic(sample, D, st, apply_polarization=True, spherical_decay=True,
                                        return_double=True)
    scale = np.abs(one).max()
    assert np.abs(got - ref).max() <= 1e-4 * scale
    assert ((got == 0) == (ref == 0)).all()
