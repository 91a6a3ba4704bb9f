"""The plane fit launched on one stream and read on another."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import engine

pytestmark = pytest.mark.gpu


def test_fit_of_another_stream_is_waited_for(cuda):
    y, z = (np.arange(40) - 20) * 55e-6, (np.arange(30) - 15) * 55e-6
    Z, Y = np.meshgrid(z, y, indexing="ij")
    phys = engine.physics(5.0e10)
    xyz = np.stack([np.full(Y.size, 0.5), Y.ravel(), Z.ravel()])
    want = engine.Pixels(xyz, 40, 30, phys, device=cuda).plane_fit()[1]
    pix = engine.Pixels(xyz, 40, 30, phys, device=cuda)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        torch.cuda._sleep(50_000_000)           # some 25 ms before the fit
        pix.start_plane_fit()
    assert np.array_equal(pix.plane_fit()[1], want)
    assert pix.plane_grid(5.0e10, 1e-6) and pix.may_be_plane(5.0e10, 1e-6)
