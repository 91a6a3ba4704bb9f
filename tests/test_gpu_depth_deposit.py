"""The column deposit (mk_beam_column_sums) against its FP64 formula in NumPy,
atoms on cell edges, on the grid's edges and off it among them.

Tolerance: a term carries the rounding of two weights, their product and the
factor's (4 x 6e-8), and a cell's at most 150 terms as many additions: 1e-5 of
the sum of the terms (all positive)."""
import ctypes

import numpy as np
import pytest
import torch

from mosaic_gb300 import _lib, engine

pytestmark = pytest.mark.gpu


def _tsc(d):
    return np.where(d <= 0.5, 0.75 - d * d, np.where(d <= 1.5, 0.5 * (1.5 - d) ** 2, 0.0)).astype(np.float32)


@pytest.mark.parametrize("ny, nz, du, dv", [(37, 20, 4.0, 1.3), (1, 9, 2.0, 0.7), (256, 3, 0.1, 11.0)])
def test_deposit_matches_the_formula(cuda, ny, nz, du, dv):
    rng = np.random.default_rng(6)
    n = 4 * ny * nz + 300
    uc, vc = (ny - 1) / 2, (nz - 1) / 2
    y = (rng.uniform(-0.6, ny - 0.4, n) - uc) * du
    z = (rng.uniform(-0.6, nz - 0.4, n) - vc) * dv
    y[:100] = (rng.integers(0, 2 * ny, 100) / 2 - uc) * du          # cells' centres and edges
    z[50:150] = (rng.integers(0, 2 * nz, 100) / 2 - vc) * dv
    y[150:160], z[160:170] = -uc * du, (nz - 1 - vc) * dv           # the grid's own edges
    y[170:180] = np.nextafter(np.float32(-uc * du), np.float32(-1e9))
    pos_A = np.stack([np.zeros(n), y, z], 1).astype(np.float32)
    sp = rng.integers(0, 2, n).astype(np.int32)
    fwd = rng.uniform(1, 30, (2, 2)).astype(np.float32)
    pos = torch.tensor(pos_A.astype(np.float64) / 1e10, device=cuda)
    spd, fd = torch.tensor(sp, device=cuda), torch.tensor(fwd, device=cuda)
    sr, si = torch.empty((ny, nz), device=cuda), torch.empty((ny, nz), device=cuda)
    grid = np.array([du, dv, uc, vc])
    engine.check(_lib.load().mk_beam_column_sums(
        n, pos.data_ptr(), spd.data_ptr(), fd.data_ptr(), 2, ny, nz,
        grid.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), sr.data_ptr(), si.data_ptr(), engine._stream_handle()))
    iu, iv = pos_A[:, 1].astype(np.float64) / du + uc, pos_A[:, 2].astype(np.float64) / dv + vc
    inside = (iu >= 0) & (iu <= ny - 1) & (iv >= 0) & (iv <= nz - 1)
    ic, jc = np.floor(iu + 0.5).astype(int), np.floor(iv + 0.5).astype(int)
    ref = np.zeros((2, ny, nz))
    for dx in (-1, 0, 1):
        for dz in (-1, 0, 1):
            ii, jj = ic + dx, jc + dz
            w = _tsc(np.abs(iu - ii)) * _tsc(np.abs(iv - jj))
            on = inside & (ii >= 0) & (ii < ny) & (jj >= 0) & (jj < nz)
            for c in range(2):
                np.add.at(ref[c], (ii[on], jj[on]), (fwd[sp, c] * w).astype(np.float64)[on])
    for got, r in ((sr, ref[0]), (si, ref[1])):
        d = np.abs(got.cpu().numpy() - r)
        assert (d <= 1e-5 * r).all(), (d / np.maximum(r, 1e-30)).max()
