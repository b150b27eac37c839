"""The NGenIC fill on grids whose columns are shared by 16, 8, 4, 2 and 1 warps,
odd counts of columns and partial blocks of the stream among them.

Tolerance: |z| <= sqrt(48 ln 2) < 6; a few units in the last place of it in
double, and in float the FP32 form's bar of the noise tests.
"""
import numpy as np
import pytest

from test_gpu_parity import Case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 20, 32, 44, 60, 64, 96, 100, 132])
def test_noise_matches_oracle(mfxlib, engine, oracle, n):
    c = Case(mfxlib, n, 100.0, 49.0, 1, 4711)
    want = oracle.ngenic_fill(n, c.seeds)
    for prec, tol in ((mfxlib.FP64, 4e-15), (mfxlib.FP32C, 4e-6)):
        j = c.job(mfxlib, engine, precision=prec, want_particles=False)
        j.run_noise(True)
        got = j.field(mfxlib.FIELD_NOISE)
        j.close()
        assert np.max(np.abs(got - want)) < tol
        assert np.array_equal(got == 0, want == 0)

