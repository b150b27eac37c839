"""FP32 form, simple cubic lattice: the assembly's x pass by component groups,
kept in shared memory and in halves, with the phase factors split by axis.

Tolerance: the forms differ in the order of FP32 roundings only, a few 2^-24 of
a displacement that is below the spacing (the bars of the fused-route tests).
"""
import numpy as np
import pytest

from test_gpu_parity import Case, rel_l2

pytestmark = pytest.mark.gpu


# 256: groups by default; 384: kept; halves from 768 (forced here)
@pytest.mark.parametrize("n,order", [(256, 2), (384, 2), (384, 3)])
def test_simple_cubic_forms_agree(mfxlib, engine, n, order, monkeypatch):
    c = Case(mfxlib, n, 300.0, 24.0, order, 77)
    out = []
    for env in ({}, {"MFX_FA_HALVES": "1"}, {"MFX_FA_XONLY": "0"}):
        for k in ("MFX_FA_HALVES", "MFX_FA_XONLY"):
            monkeypatch.delenv(k, raising=False)
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        j = c.job(mfxlib, engine, precision=mfxlib.FP32C, vel64=False)
        j.run()
        out.append(j.particles())
        j.close()
    for pos, vel, ids in out[1:]:
        assert np.sqrt(np.mean(((pos - out[0][0]) * n / c.L) ** 2)) < 1e-6
        assert rel_l2(vel.astype(np.float64), out[0][1].astype(np.float64)) < 5e-6
        assert np.array_equal(ids, out[0][2])


def test_simple_cubic_second_lattice_matches_fp64(mfxlib, engine):
    """The secondary lattice's shift: x factor in the x pass, y and z factors in
    the y pass."""
    c = Case(mfxlib, 32, 300.0, 24.0, 2, 5)
    got = []
    for prec in (mfxlib.FP32C, mfxlib.FP64):
        j = c.job(mfxlib, engine, precision=prec)
        j.run()
        j.set_species(secondary=True, id_offset=1, c_species=0.85, mass_factor=0.045)
        j.assemble(3)
        got.append(j.particles())
        j.close()
    (p32, v32, i32), (p64, v64, i64) = got
    assert np.sqrt(np.mean(((p32 - p64) * c.n / c.L) ** 2)) < 1e-5
    assert rel_l2(v32, v64) < 1e-5
    assert np.array_equal(i32, i64)
