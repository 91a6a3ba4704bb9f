"""Where the FP64 sum's expansion of the scattering factors would lose more than
it states -- high energies near forward with atoms along the beam, wide electron
clouds, a factor that anomalous scattering cancels, very large Debye-Waller
factors -- every factor is evaluated per term: against the same kernel under an
analyser that accepts every direction, which selects that path and multiplies by
exactly 1.

Tolerance: 2e-12 of the sum of |E| |F| (the stated bound of a term) plus 4e-16 of
that of |E| times the uncancelled factor (the rounding of f0 + f' itself)."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import engine
from mosaic_gb300.tables import ScatteringTables

pytestmark = pytest.mark.gpu
K10 = 2 * np.pi / 1.2398e-10          # wave number at 10 keV


def _f0(wk, s):
    return wk[5] + sum(wk[i] * np.exp(-wk[6 + i] * s * s) for i in range(5))


@pytest.mark.parametrize("species, kev, tt, cancel, dw", [
    ("K", 100.0, 0.2, None, 0.0), ("H1-", 100.0, 0.2, None, 0.0), ("Cs", 100.0, 0.5, None, 0.0),
    ("H1-", 60.0, 0.3, None, 0.0), ("K", 60.0, 2.0, None, 0.0), ("H1-", 30.0, 1.0, None, 0.0),
    ("Cu", 10.0, 40.0, 1e-3, 0.0), ("Cu", 10.0, 40.0, 1e-4, 0.0), ("K", 10.0, 25.0, 3e-4, 0.0),
    ("Cu", 60.0, 2.0, None, 900.0), ("Cu", 10.0, 25.0, None, 3000.0),
    ("Cu", 10.0, 25.0, None, 0.5), ("K", 20.0, 10.0, None, 0.0),
])
@pytest.mark.parametrize("along", [0, 2])
def test_a_term_stays_within_its_bound(cuda, species, kev, tt, cancel, dw, along):
    wk = np.asarray(ScatteringTables().f0[species], np.float64).ravel()[:11].astype(np.float32)
    k, R = K10 * kev / 10.0, 0.7
    rng = np.random.default_rng(3)
    rot = np.radians(tt)
    M = np.array([[np.cos(rot), 0, -np.sin(rot)], [0, 1, 0], [np.sin(rot), 0, np.cos(rot)]])
    y = (np.arange(3) - 1) * 5e-6
    Z, Y = np.meshgrid(y, y, indexing="ij")
    xyz = M @ np.stack([np.full(9, R), Y.ravel(), Z.ravel()])
    s = k * 1e-10 / (4 * np.pi) * 2 * np.sin(rot / 2)
    F0 = _f0(wk.astype(float), s)
    F = F0 if cancel is None else cancel * F0
    worst = 0.0
    for trial in range(12):
        pos = np.zeros((6, 3))
        pos[:, along] = 1.49e-7 * R * (1.0 - 0.02 * rng.random(6))
        table = engine.SpeciesTable([species], wk[None], np.array([_f0(wk, 0.0)], np.float32),
                                    np.array([F - F0 + 0j]))
        if dw:
            table.dw_b = np.array([dw], np.float32)
        amp = np.zeros((6, 2), np.float32)
        amp[:, 0] = rng.uniform(0.5, 1.0, 6)
        atoms = engine.Atoms(torch.tensor(pos, device=cuda), torch.zeros(6, dtype=torch.int32, device=cuda),
                             torch.tensor(amp, device=cuda), np.array([6]), table)
        out = []
        for analyser in (None, (1, M[:, 0], np.pi, 0.0)):
            phys = engine.physics(k, analyser=analyser)
            pix = engine.Pixels(xyz, 3, 3, phys, device=cuda)
            out.append(engine.run_plain(atoms, pix, phys).cpu().numpy())
        decay = np.exp(-dw * s * s)
        scale = engine.R_E * float(amp.sum()) * decay
        worst = max(worst, np.abs(out[0] - out[1]).max() / (scale * (2e-12 * abs(F) + 4e-16 * F0)))
    assert worst <= 1.0, worst
