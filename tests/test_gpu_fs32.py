"""FP32 form without fused transforms: the pruned single-precision passes
against the cuFFT route of the same form and against the plain FP64 form.

Tolerances: those of the fused route's comparison with cuFFT (both FP32).
"""
import numpy as np
import pytest

from test_gpu_parity import Case, rel_l2

pytestmark = pytest.mark.gpu


def fields_of(mfx, j, order):
    ids = [mfx.FIELD_PHI1] + ([mfx.FIELD_PHI2] if order > 1 else [])
    if order > 2:
        ids += [mfx.FIELD_PHI3, mfx.FIELD_A3X, mfx.FIELD_A3Y, mfx.FIELD_A3Z]
    return [j.field(f) for f in ids]


# run-time radices 2 .. 16 (padded lengths 18, 30, 42, 54, 90, 150, 168, 210, 300),
# MUSIC1's filled Nyquist planes at the instances 24 .. 384, 1LPT at grid lengths
@pytest.mark.parametrize("n,order,lattice,music", [
    (12, 3, 0, False), (20, 3, 1, False), (28, 3, 2, False), (36, 2, 0, False), (60, 3, 1, False), (100, 3, 1, False),
    (112, 2, 0, False), (140, 2, 0, False), (200, 2, 1, False), (16, 3, 2, True), (32, 3, 1, True), (64, 3, 2, True),
    (128, 3, 1, True), (256, 2, 0, True), (48, 1, 2, False), (72, 1, 1, False), (192, 1, 0, False), (32, 1, 2, True)])
def test_matches_cufft_route(mfxlib, engine, n, order, lattice, music, monkeypatch):
    c = Case(mfxlib, n, 300.0, 24.0, order, 77, lattice=lattice)
    kw = dict(noise_generator=mfxlib.NOISE_MUSIC1, music_seed=77) if music else {}
    out = []
    for env in ("1", "0"):
        monkeypatch.setenv("MFX_FUSED", env)
        j = c.job(mfxlib, engine, precision=mfxlib.FP32C, **kw)
        j.run()
        assert (j.launch_count()[1] == int(music)) == (env == "1")
        out.append((fields_of(mfxlib, j, order), j.particles()))
        j.close()
    for a, b in zip(out[0][0], out[1][0]):
        assert rel_l2(a, b) < 5e-6
    (p0, v0, i0), (p1, v1, i1) = out[0][1], out[1][1]
    delta = c.L / (c.n * 2 ** (lattice / 3.0))
    assert np.sqrt(np.mean(((p0 - p1) / delta) ** 2)) < 1e-6
    assert rel_l2(v0.astype(np.float64), v1.astype(np.float64)) < 5e-6
    assert np.array_equal(i0, i1)


@pytest.mark.parametrize("box", [1.0, 1.0e5])
def test_extreme_boxes_stay_in_range(mfxlib, engine, box):
    """Products of three Hessians at the ends of the box sizes: finite, and the
    plain FP64 form's potentials."""
    c = Case(mfxlib, 20, box, 24.0, 3, 9)
    got = []
    for prec in (mfxlib.FP32C, mfxlib.FP64):
        j = c.job(mfxlib, engine, precision=prec)
        j.run()
        got.append(fields_of(mfxlib, j, 3))
        j.close()
    for a, b in zip(*got):
        assert np.isfinite(a).all() and rel_l2(a, b) < 1e-5
