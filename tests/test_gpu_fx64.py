"""The plain FP64 form's fixed-point transforms: every radix and edge of the
lengths they take, against the oracle and against the cuFFT route.

Tolerance: a transform's error is below 2^-52 of its output's norm (the last
bits of 62-bit integers against the norm of at most 2^11 of them), a potential
passes through at most 15 of them, a product of two Hessians up to four times
as sensitive as its factors, and the reference transforms err by as much: 3e-14.
"""
import numpy as np
import pytest

from test_gpu_parity import Case, rel_l2

pytestmark = pytest.mark.gpu

TOL = 3e-14


def fields_of(mfx, j, order):
    ids = [mfx.FIELD_PHI1, mfx.FIELD_PHI2]
    if order > 2:
        ids += [mfx.FIELD_PHI3, mfx.FIELD_A3X, mfx.FIELD_A3Y, mfx.FIELD_A3Z]
    return [j.field(f) for f in ids]


# padded lengths 12 = 3*4 .. 90 = 9*10: the run-time radices 2, 3, 4, 5, 6, 7, 9,
# 10 and the instances of 16, 24, 32, 48, 64, 72 and 96
@pytest.mark.parametrize("n,lattice", [(8, 0), (12, 1), (16, 2), (20, 0), (28, 1), (32, 1), (36, 0), (40, 2), (48, 1),
                                       (60, 0), (64, 2)])
def test_lengths_match_oracle(mfxlib, engine, oracle, n, lattice):
    c = Case(mfxlib, n, 100.0, 24.0, 3, 99, lattice=lattice)
    j = c.job(mfxlib, engine)
    j.run()
    assert j.launch_count()[1] == 0  # no FFT library call
    res = c.oracle(oracle)
    got = fields_of(mfxlib, j, 3)
    want = [res["phi"], res["phi2"], res["phi3"]] + res["A3"]
    scale = [c.coef["g1"], c.coef["g2"], c.coef["g3"]] + 3 * [c.coef["g3c"]]
    for a, b, s in zip(got, want, scale):
        assert rel_l2(a * s, b) < TOL
    pos, vel, ids = j.particles()
    assert rel_l2(vel, res["vel"]) < TOL
    assert rel_l2(pos, res["pos"]) < 1e-15
    assert np.array_equal(ids, res["ids"])
    j.close()


# 84, 100, 112, 120, 140, 180, 200: padded lengths with factors 5, 7 and 9; the
# others the instances of 144 .. 384 (and N-grid lengths 96 .. 256)
@pytest.mark.parametrize("n,order,music", [(84, 3, False), (96, 3, False), (100, 3, False), (112, 2, False),
                                           (120, 3, False), (128, 3, True), (140, 2, False), (180, 2, False),
                                           (192, 3, False), (200, 2, False), (256, 2, True)])
def test_lengths_match_cufft_route(mfxlib, engine, n, order, music, monkeypatch):
    c = Case(mfxlib, n, 300.0, 24.0, order, 5, lattice=1)
    kw = dict(noise_generator=mfxlib.NOISE_MUSIC1, music_seed=77) if music else {}
    out = []
    for env in ("1", "0"):
        monkeypatch.setenv("MFX_FUSED", env)
        j = c.job(mfxlib, engine, **kw)
        j.run()
        assert (j.launch_count()[1] == int(music)) == (env == "1")
        out.append(fields_of(mfxlib, j, order) + list(j.particles()))
        j.close()
    for a, b in zip(out[0][:-3], out[1][:-3]):
        assert rel_l2(a, b) < TOL
    assert rel_l2(out[0][-2], out[1][-2]) < TOL
    assert rel_l2(out[0][-3], out[1][-3]) < 1e-15
    assert np.array_equal(out[0][-1], out[1][-1])


def test_other_lengths_take_cufft(mfxlib, engine, oracle):
    c = Case(mfxlib, 44, 100.0, 24.0, 2, 3)  # 66 = 2 * 3 * 11
    j = c.job(mfxlib, engine)
    j.run()
    assert j.launch_count()[1] > 0
    assert rel_l2(j.particles()[1], c.oracle(oracle)["vel"]) < TOL
    j.close()


def test_scale_of_the_field_does_not_matter(mfxlib, engine):
    """One exponent per pencil: a field times a power of two gives the same
    bits, times that power (phi2: its square)."""
    c = Case(mfxlib, 48, 100.0, 24.0, 2, 8)
    out = []
    for s in (0, -200, 200):
        c.amp *= 2.0 ** s
        j = c.job(mfxlib, engine)
        j.run()
        out.append((j.field(mfxlib.FIELD_PHI1) * 2.0 ** -s, j.field(mfxlib.FIELD_PHI2) * 2.0 ** (-2 * s)))
        j.close()
        c.amp *= 2.0 ** -s
    for a in out[1:]:
        assert np.array_equal(a[0], out[0][0]) and np.array_equal(a[1], out[0][1])


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_input_stays_visible(mfxlib, engine, bad):
    n = 20
    c = Case(mfxlib, n, 100.0, 24.0, 2, 8)
    f = np.random.default_rng(3).standard_normal((n, n, n))
    f[3, 4, 5] = bad
    j = mfxlib.Job(engine, n, c.L, 2, None, c.amp, c.coef, noise_field=f, lunit=c.lunit, vunit=c.vunit)
    j.run()
    pos, vel, _ = j.particles()
    assert not np.isfinite(pos).any() and not np.isfinite(vel).any()
    j.close()


def test_zero_field_gives_the_lattice(mfxlib, engine):
    n = 24
    c = Case(mfxlib, n, 100.0, 24.0, 3, 8)
    j = mfxlib.Job(engine, n, c.L, 3, None, c.amp, c.coef, noise_field=np.zeros((n, n, n)), lunit=c.lunit,
                   vunit=c.vunit)
    j.run()
    pos, vel, _ = j.particles()
    q = np.arange(n) / float(n) * c.lunit
    want = np.stack(np.meshgrid(q, q, q, indexing="ij"), -1).reshape(-1, 3)
    assert np.array_equal(pos, want) and not vel.any()
    j.close()


# every further instance: both forms against cuFFT, order 3 where it is quick
@pytest.mark.parametrize("n", [56, 60, 72, 80, 84, 100, 108, 112, 120, 140, 144, 160, 168, 180, 196, 200, 216, 224,
                               240, 252])
def test_further_instances_match_cufft_route(mfxlib, engine, n, monkeypatch):
    order = 3 if n <= 144 else 2
    c = Case(mfxlib, n, 300.0, 24.0, order, 6, lattice=1)
    for prec, tol in ((mfxlib.FP64, TOL), (mfxlib.FP32C, 5e-6)):
        out = []
        for env in ("1", "0"):
            monkeypatch.setenv("MFX_FUSED", env)
            j = c.job(mfxlib, engine, precision=prec)
            j.run()
            out.append(fields_of(mfxlib, j, order) + [j.particles()[1].astype(np.float64)])
            j.close()
        for a, b in zip(*out):
            assert rel_l2(a, b) < tol
