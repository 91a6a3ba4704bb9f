"""Staging kernels against plain PyTorch/NumPy: the metre positions to the
bit, species indices and counts, and the tile build's order (every atom in
one tile, tiles compact) where its keys change length."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import engine
from mosaic_gb300.tables import ScatteringTables

pytestmark = pytest.mark.gpu


def _table(n):
    return engine.SpeciesTable.build(["Cu", "Ni", "Na", "Cl"][:n], ScatteringTables(), 10000.0)


def test_positions_in_metres_are_the_rounded_quotient(cuda):
    rng = np.random.default_rng(0)
    x = np.concatenate([rng.uniform(-1e4, 1e4, 300000), 10.0 ** rng.uniform(-30, 30, 300000),
                        np.arange(-4096, 4096) / 64.0, [0.0]]).astype(np.float32)
    x = np.resize(x, (x.size // 3 * 3,)).reshape(-1, 3)
    a = engine.atoms_lab(x, np.zeros(len(x), np.int32), np.eye(3), np.zeros(3), _table(1), device=cuda)
    assert torch.equal(a.pos.cpu(), torch.from_numpy(x.astype(np.float64) / 1e10))


@pytest.mark.parametrize("n", [1, 31, 256, 1025, 400003])
@pytest.mark.parametrize("n_species", [1, 3, 16])
def test_species_index(cuda, n, n_species):
    rng = np.random.default_rng(n)
    codes = rng.integers(0, n_species, n).astype(np.uint8)
    lut = rng.permutation(n_species).astype(np.int32)
    out = torch.full((n,), -7, dtype=torch.int32, device=cuda)
    counts = torch.zeros(16, dtype=torch.int64, device=cuda)
    engine.species_index(torch.from_numpy(codes).to(cuda), lut, n_species, out, counts)
    assert np.array_equal(out.cpu().numpy(), lut[codes])
    assert np.array_equal(counts.cpu().numpy(), np.bincount(lut[codes], minlength=16))
    if n_species == 3 and n > 1000:     # a code without an entry is not counted
        engine.species_index(torch.from_numpy(codes).to(cuda), lut[:2] % 2, 2, out, counts)
        assert int(counts.sum()) == n + int((codes < 2).sum())


@pytest.mark.parametrize("n, box", [(700, (30, 30, 30)), (1 << 17, (200, 200, 200)),
                                    ((1 << 17) + 1, (200, 200, 200)), (200000, (4000, 60, 50)),
                                    (5000, (300, 0, 0))])
def test_tiles_hold_every_atom_and_stay_compact(cuda, n, box):
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 3)) * np.array(box)).astype(np.float32)
    sp = rng.integers(0, 2, n).astype(np.int32)
    atoms = engine.atoms_lab(pos, sp, np.eye(3), np.zeros(3), _table(2), device=cuda)
    k, T = 5e10, 128
    t = engine.Tiles(atoms, k, T, device=cuda)
    o = t.origin.cpu().numpy()
    p4 = t.pos.cpu().numpy().reshape(t.n_tiles, T // 2, 4, 2)        # x0 x1 y0 y1 z0 z1 w0 w1
    amp = t.amp.cpu().numpy().reshape(t.n_tiles, T // 2, 2, 2)
    live = amp[:, :, 0, :] != 0
    got = o[:, None, None, :3] + np.moveaxis(p4[:, :, :3, :], 2, 3) / (k / (2 * np.pi))
    want = atoms.pos.cpu().numpy()
    assert live.sum() == n
    a, b = np.sort(got[live][:, 0]), np.sort(want[:, 0])
    assert np.abs(a - b).max() <= 1e-15         # float32 offsets of a few hundred A
    # a tile's box against the sample's share of the volume (or length)
    dims = np.array([b for b in box if b > 0], float)
    share = (np.prod(dims) * T / (n / 2)) ** (1 / len(dims)) * 1e-10
    assert np.median(o[:, 3]) <= 1.5 * share


@pytest.mark.parametrize("shapes", [[(5, 3)], [(1, 7), (33, 9), (7, 1), (16, 16)]])
def test_scan_pixels_match_numpy(cuda, shapes):
    """Frames into the sample frame and their prologue, against NumPy and the
    single-exposure prologue; the frames of one ROI may share their array."""
    from mosaic_gb300 import workloads
    from mosaic_gb300.scan import Frame
    rng = np.random.default_rng(7)
    frames, bd = [], []
    for i, (ny, nz) in enumerate(shapes + shapes[:1]):
        R = workloads.random_rotations(1, rng)[0].astype(np.float32)
        t = rng.uniform(-500, 500, 3).astype(np.float32)
        P = frames[0].pixels if i == len(shapes) else rng.uniform(0.5e10, 1.5e10, (3, ny * nz))
        frames.append(Frame(R, t, P, (ny, nz)))
        bd.append(R.astype(np.float64).T @ np.array([1.0, 0, 0]))
    phys = engine.physics(5.0e10)
    px = engine.Pixels.of_scan(frames, np.array(bd), phys, device=cuda)
    for (off, m), f, b in zip(px.spans, frames, bd):
        R = np.asarray(f.rotation, np.float64)
        want = (R.T @ (f.pixels - np.asarray(f.translation, np.float64)[:, None]) / 1e10).T
        got = px.xyz[off:off + m].cpu().numpy()
        # three products and two sums, in whatever order and contraction
        assert np.abs(got - want).max() <= 4 * np.finfo(float).eps * np.abs(f.pixels).max() / 1e10 * 3
        ph = engine.physics(5.0e10, beam_dir=b)
        one = engine.Pixels(np.ascontiguousarray(got.T), *f.shape, ph, device=cuda)
        for a, c in ((px.r0, one.r0), (px.q, one.q), (px.u, one.u), (px.phasor, one.phasor)):
            assert torch.equal(a[off:off + m], c)
