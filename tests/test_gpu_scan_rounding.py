"""A scan's pixel positions to the bit: R^T (P - t) as its first product, then
one fused multiply-add each (what NumPy's matrix product gives), divided by 1e10
-- an ulp of a position is ~1e-5 rad of a frame's phase."""
from fractions import Fraction

import numpy as np
import pytest

from mosaic_gb300 import engine, workloads
from mosaic_gb300.scan import Frame

pytestmark = pytest.mark.gpu


def _fma(a, b, c):
    return float(Fraction(float(a)) * Fraction(float(b)) + Fraction(float(c)))


@pytest.mark.parametrize("ny, nz", [(1, 1), (5, 3), (64, 16)])
def test_positions_are_the_rounded_chain(cuda, ny, nz):
    rng = np.random.default_rng(ny)
    frames, bd = [], []
    for _ in range(3):
        R = workloads.random_rotations(1, rng)[0].astype(np.float32)
        t = rng.uniform(-500, 500, 3).astype(np.float32)
        frames.append(Frame(R, t, rng.uniform(-1e10, 1e10, (3, ny * nz)), (ny, nz)))
        bd.append(R.astype(np.float64).T @ np.array([1.0, 0, 0]))
    px = engine.Pixels.of_scan(frames, np.array(bd), engine.physics(5.0e10), device=cuda)
    for (off, m), f in zip(px.spans, frames):
        R, d = f.rotation.astype(np.float64), f.pixels - f.translation.astype(np.float64)[:, None]
        want = np.array([[_fma(R[2, c], d[2, i], _fma(R[1, c], d[1, i], R[0, c] * d[0, i])) / 1e10
                          for c in range(3)] for i in range(m)])
        assert np.array_equal(px.xyz[off:off + m].cpu().numpy(), want)
