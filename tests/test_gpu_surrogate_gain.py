"""What the scan surrogate's times are measured against: the exact-only scan in
the form a user gets, and the direct sum under a name of its own, the same in
either mode of the run.

Tolerance of the exact scan against the direct sum: 1e-4 of the peak, the FP32
forms'."""
import numpy as np
import pytest

from mosaic_gb300 import workloads
from mosaic_gb300.surrogate import SurrogateScan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exact_all", [True, False])
def test_gains_are_against_what_they_say(cuda, monkeypatch, exact_all):
    w = workloads.cu_bumps_scan_4m(cells=24, npix=64)
    off = np.radians(np.linspace(-0.1, 0.1, 11))
    sc = SurrogateScan(w.beam, w.sample, w.detector, w.stage, off, off.copy(), roi=64, stride=3, fit_steps=50,
                       sc_kwargs=w.sc_kwargs)
    calls, exact = [], sc.exact

    def spy(idx, *a, direct=False, **k):
        calls.append((len(idx), direct))
        return exact(idx, *a, direct=direct, **k)
    monkeypatch.setattr(sc, "exact", spy)
    res = sc.run(exact_all=exact_all)
    n = 121
    # the whole scan only in the form every caller gets, the direct sum on a sample
    assert ((n, False) in calls) == exact_all and (n, True) not in calls
    assert (sc.DIRECT_FRAMES, True) in calls
    assert res["gain_vs_exact"] == pytest.approx(res["exact_seconds"] / res["seconds"])
    assert res["gain"] == pytest.approx(res["direct_seconds"] / res["seconds"])
    assert res["exact_frames_per_s"] == pytest.approx(n / res["exact_seconds"])
    if exact_all:
        assert res["direct_err"].shape == (sc.DIRECT_FRAMES,) and res["direct_err"].max() <= 1e-4
        assert res["final_err"].shape == (n,)
