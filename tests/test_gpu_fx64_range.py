"""Range and precision of the plain FP64 form's fixed-point transforms, where a
field is as far from a Gaussian one as a caller can make it.

Tolerance: that of the other route comparisons (test_gpu_fx64.py).
"""
import numpy as np
import pytest

from test_gpu_parity import Case, rel_l2

pytestmark = pytest.mark.gpu

TOL = 3e-14


# sizes of the N-grid and padded lengths whose sums have the least head room
@pytest.mark.parametrize("n", [40, 48, 60, 72, 96, 120, 140, 160, 180])
def test_sheets_match_cufft_route(mfxlib, engine, n, monkeypatch):
    """A sheet in x times a phase in z, all amplitudes one: every x pencil holds
    one value, the largest sum a transform can make of its largest element.  The
    sixteen field amplitudes pass that value through all mantissas."""
    c = Case(mfxlib, n, 100.0, 24.0, 1, 3)
    amp = np.ones_like(c.amp)
    z = np.arange(n)
    got = []
    for env in ("1", "0"):
        monkeypatch.setenv("MFX_FUSED", env)
        out = []
        for phase in (0.25, 0.75):
            for step in range(16):
                f = np.zeros((n, n, n))
                f[0] = 2.0 ** (step / 16.0) * np.cos(2.0 * np.pi * 3 * z / n + np.pi * phase)
                j = mfxlib.Job(engine, n, c.L, 1, None, amp, c.coef, noise_field=f, lunit=c.lunit, vunit=c.vunit)
                j.run()
                out.append(j.particles()[1])
                j.close()
        got.append(out)
    for a, b in zip(*got):
        assert rel_l2(a, b) < TOL
