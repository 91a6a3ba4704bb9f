"""The column pass on the field's rows only (mk_prop_cols_rows) against the
same pass on the whole padded grid: the rows it forms itself (edges repeated,
or a constant) and the ones it leaves out, at every last radix (2, 4, 8), one
to sixteen columns a block and fields that fill the grid or a single row.

Tolerance: the two differ by the row transforms' rounding of repeated rows
(none: they are the same rows) and, for a constant, of one bin: 1e-6 of max."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import _lib, engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("ny2, nz2, nz, z0", [
    (4, 2, 1, 1), (8, 8, 5, 2), (1, 16, 9, 3), (2, 32, 32, 0), (32, 64, 1, 63), (64, 128, 100, 14),
    (16, 1024, 700, 162), (8, 2048, 1500, 274), (8, 4096, 2500, 798), (4, 8192, 5000, 0)])
def test_rows_match_the_padded_grid(cuda, ny2, nz2, nz, z0, mode):
    L = _lib.load()
    g = torch.Generator(device=cuda)
    g.manual_seed(nz2 + nz)
    E = torch.randn((nz, ny2, 2), generator=g, device=cuda)
    E = torch.view_as_complex(E)
    c = 0.4 - 1.3j
    idx = torch.arange(nz2, device=cuda) - z0
    full = E[idx.clamp(0, nz - 1)]
    if mode:
        full[(idx < 0) | (idx >= nz)] = c
    k = 2 * np.pi / 1.2398e-10
    ws_n = int(L.mk_prop_cols_workspace_size(ny2, nz2))
    ws = torch.empty(ws_n, dtype=torch.uint8, device=cuda)
    args = (2e-6, 3e-6, k, 0.04, k, 0.0, 0.0, ws.data_ptr(), ws_n, engine._stream_handle())
    A, B = torch.fft.fft(full.contiguous(), dim=-1), torch.fft.fft(E.contiguous(), dim=-1)
    _lib.check(L.mk_prop_cols(A.data_ptr(), ny2, nz2, *args))
    _lib.check(L.mk_prop_cols_rows(B.data_ptr(), ny2, nz2, z0, nz, mode, c.real, c.imag, *args))
    engine.sync()
    ref = A[z0:z0 + nz]
    assert float((B - ref).abs().max() / ref.abs().max()) <= 1e-6
