"""The FP64 sum's expansion of the direction-dependent factors about each
pixel's direction, against the same kernel with every factor evaluated per
term (an analyser that accepts every direction selects that path and
multiplies by exactly 1).

Tolerance 2e-12 of the largest term sum: the remainders and the FP32 change
stay below 2e-13 per term at 10 keV (b ~ 1/s^2), with a factor ten to spare."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import engine
from mosaic_gb300.tables import ScatteringTables

pytestmark = pytest.mark.gpu


def _atoms(cuda, half, n, dw, real):
    rng = np.random.default_rng(4)
    pos = rng.uniform(-half, half, (n, 3)) / np.sqrt(3.0)
    pos[0] = [half, 0, 0]
    sp = rng.integers(0, 3, n).astype(np.int32)
    table = engine.SpeciesTable.build(["Cu", "Na", "Cl"], ScatteringTables(), 10000.0, dw)
    amp = rng.uniform(-1, 1, (n, 2)).astype(np.float32)
    if real:                                # no imaginary part in any staging step
        amp[:, 1] = 0.0
    return engine.Atoms(torch.tensor(pos, device=cuda), torch.tensor(sp, device=cuda),
                        torch.tensor(amp, device=cuda), np.bincount(sp, minlength=3).astype(np.int64), table)


@pytest.mark.parametrize("excursion", [1e-9, 6e-8, 1.49e-7, 1.51e-7, 1e-5])
@pytest.mark.parametrize("flags", [
    dict(), dict(real=True), dict(apply_pol=True, pol=(1.0, 0.0, 1.0, 0.0), spherical_decay=True),
    dict(apply_pol=True, pol=(0.6, 0.0, 0.6, 0.8), spherical_decay=True, dw=True),
    dict(apply_pol=True, pol=(1.0, 0.0, 0.0, 1.0), tt=80.0, spherical_decay=True),     # P_pol ~ 0.03
    dict(remove_forward=True, tt=0.0, dw=True), dict(tt=0.0, remove_forward=True, n_pix=(1, 1)),
])
def test_expansion_matches_the_per_term_factors(cuda, excursion, flags):
    f = dict(flags)
    tt, dw, (ny, nz) = np.radians(f.pop("tt", 25.0)), f.pop("dw", False), f.pop("n_pix", (19, 13))
    k, R = 2 * np.pi / 1.2398e-10, 0.7
    atoms = _atoms(cuda, excursion * R, 700, {"Cu": 0.55, "Cl": 1.3} if dw else None, f.pop("real", False))
    y, z = (np.arange(ny) - (ny - 1) / 2) * 55e-6, (np.arange(nz) - (nz - 1) / 2) * 55e-6
    Z, Y = np.meshgrid(z, y, indexing="ij")
    rot = np.array([[np.cos(tt), 0, -np.sin(tt)], [0, 1, 0], [np.sin(tt), 0, np.cos(tt)]])
    xyz = rot @ np.stack([np.full(Y.size, R), Y.ravel(), Z.ravel()])
    out = []
    for analyser in (None, (1, rot[:, 0], np.pi, 0.0)):
        phys = engine.physics(k, analyser=analyser, **f)
        pix = engine.Pixels(xyz, ny, nz, phys, device=cuda)
        out.append(engine.run_plain(atoms, pix, phys).cpu().numpy())
    scale = engine.R_E * float(np.abs(atoms.amp.cpu().numpy()).sum()) * 29.0
    assert np.isfinite(out[0]).all()
    assert np.abs(out[0] - out[1]).max() <= 2e-12 * scale, np.abs(out[0] - out[1]).max() / scale
