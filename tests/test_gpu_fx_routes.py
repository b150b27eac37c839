"""The pruned transforms where other tests do not go: grids that take the
run-time kernels with three steps and 4 or 2 pencils a CTA, the instances of three
steps, and grid lengths from 384 up, in both forms, against the cuFFT route.

Tolerances: FP64: a field passes at most 15 transforms of 2.8e-16 each (the most
that an FP64 transform is off, tests/test_fx64_range.py), 1.1e-15 if they are
independent, and a product of Hessians is up to four times as sensitive as they
are: 4.4e-15.  FP32: that of the other comparisons of two FP32 routes.
"""
import numpy as np
import pytest

from test_gpu_parity import Case, rel_l2

pytestmark = pytest.mark.gpu

TOL = {8: 4.4e-15, 4: 5e-6}


def outputs(mfx, c, engine, prec, order, music=False, fields=None, **kw):
    """Potentials and a sample of velocities (every grid line's start at least)."""
    if music:
        kw.update(noise_generator=mfx.NOISE_MUSIC1, music_seed=77)
    j = c.job(mfx, engine, precision=prec, **kw)
    j.run()
    ids = [mfx.FIELD_PHI2, mfx.FIELD_PHI3, mfx.FIELD_A3X, mfx.FIELD_A3Y, mfx.FIELD_A3Z][:{1: 0, 2: 1, 3: 5}[order]]
    out = [j.field(f) for f in (ids if fields is None else ids[:fields])]
    if kw.get("want_particles", True):
        count = min(j.num_particles, 1 << 21)
        for first in {0, (j.num_particles - count) // 2, j.num_particles - count}:
            vel = np.empty((count, 3), np.float64 if j.vel64 else np.float32)
            j.fetch_particles_range_into(first, count, None, vel.ctypes.data, None)
            out.append(vel.astype(np.float64))
    ffts = j.launch_count()[1]
    j.close()
    return out, ffts


def compare(mfx, engine, monkeypatch, n, order, prec, music=False, **kw):
    c = Case(mfx, n, 300.0, 24.0, order, 6, lattice=0)
    got = []
    for env in ("1", "0"):
        monkeypatch.setenv("MFX_FUSED", env)
        out, ffts = outputs(mfx, c, engine, prec, order, music, **kw)
        assert (ffts == int(music)) == (env == "1")  # MUSIC1's own transform stays with cuFFT
        got.append(out)
    for a, b in zip(*got):
        assert rel_l2(a, b) < TOL[8 if prec == mfx.FP64 else 4]


# padded lengths 420 .. 960: three steps, 4 pencils a CTA, 450, 900: 2; the grid
# lengths between 280 and 640
@pytest.mark.parametrize("n,order", [(280, 2), (288, 2), (300, 3), (320, 2), (360, 2), (400, 2), (448, 2), (480, 2),
                                     (600, 2), (640, 1)])
def test_run_time_kernels(mfxlib, engine, n, order, monkeypatch):
    compare(mfxlib, engine, monkeypatch, n, order, mfxlib.FP64)


# padded 576 (two steps), 768 and 1152 (three), grid lengths 384, 512, 768
@pytest.mark.parametrize("n,order,kw", [(384, 3, dict(fields=2)), (512, 3, dict(fields=2)), (512, 1, {}), (768, 1, {}),
                                        (768, 2, dict(want_particles=False))])
def test_large_instances(mfxlib, engine, n, order, kw, monkeypatch):
    compare(mfxlib, engine, monkeypatch, n, order, mfxlib.FP64, **kw)


# single precision: MUSIC1 at padded 768, first order at grid lengths 384 .. 768
@pytest.mark.parametrize("n,order,music", [(512, 2, True), (384, 1, False), (512, 1, False), (768, 1, False)])
def test_large_instances_single(mfxlib, engine, n, order, music, monkeypatch):
    compare(mfxlib, engine, monkeypatch, n, order, mfxlib.FP32C, music, vel64=False)


# the small grids without an instance: padded lengths 12 to 60, one and two steps
@pytest.mark.parametrize("n", [8, 12, 20, 24, 28, 36, 40])
def test_small_run_time_kernels(mfxlib, engine, n, monkeypatch):
    for prec in (mfxlib.FP64, mfxlib.FP32C):
        c = Case(mfxlib, n, 100.0, 24.0, 3, 11, lattice=1)
        got = []
        for env in ("1", "0"):
            monkeypatch.setenv("MFX_FUSED", env)
            got.append(outputs(mfxlib, c, engine, prec, 3)[0])
        for a, b in zip(*got):
            assert rel_l2(a, b) < TOL[8 if prec == mfxlib.FP64 else 4]
