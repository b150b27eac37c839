"""The fixed-point transforms' arithmetic (fx64.cuh), built for the host, for
every length and order of radices that can run, against long double transforms:
pencils made to drive its sums as high as they go, and spectra from flat to k^-4.

Tolerances, relative to the output's norm.  Spectra: the error of numpy's FP64
transform of the same pencils (the transforms replaced one).  Made pencils: the
scale keeps the largest input, or the root of the number of terms times their
rms, above 2^54 units of the result's last place, and an output carries the
roundings of at most 24 products and 3 steps, about 4 of these units: 2^-52.
"""
import pathlib
import subprocess

import numpy as np
import pytest

from monofonic_gb300 import build

HERE = pathlib.Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = tmp_path_factory.mktemp("fx64") / "fx64_check"
    subprocess.check_call([str(pathlib.Path(build._cuda_home()) / "bin" / "nvcc"), *build.ARCH, "-O2", "-std=c++17",
                           "--expt-relaxed-constexpr", "-I", str(build.PKG / "csrc"), "-o", str(exe),
                           str(HERE / "fx64_check.cu")])
    out = subprocess.run([str(exe), "list"], capture_output=True, text=True, check=True).stdout
    plans = sorted({(int(w[0]), w[1], tuple(map(int, w[2:]))) for w in map(str.split, out.splitlines())})
    return exe, plans


def run(exe, L, kind, radices, x):
    """x: [pencils][L] complex for kind s, [pencils][2][L/2 + 1] complex for c, [pencils][2][L] real for r."""
    out = subprocess.run([str(exe), "run", str(L), kind, *map(str, radices)], input=np.ascontiguousarray(x).tobytes(),
                         capture_output=True, check=True).stdout
    got = np.frombuffer(out, dtype=np.float64 if kind == "c" else np.complex128)
    return got.reshape(len(x), -1)


def transform(kind, x, L):
    """The same in numpy, in the precision of x."""
    if kind == "s":
        return np.fft.fft(x, axis=-1)
    if kind == "r":
        return np.fft.rfft(x, axis=-1).reshape(len(x), -1)
    return np.fft.irfft(x, n=L, axis=-1, norm="forward").reshape(len(x), -1)


def wide(x):
    return x.astype(np.clongdouble if np.iscomplexobj(x) else np.longdouble)


def rel(got, want):
    """Per pencil, relative to the pencil's norm."""
    d = np.sqrt(np.sum(np.abs(got - want) ** 2, axis=1).astype(np.float64))
    return d / np.sqrt(np.sum(np.abs(want) ** 2, axis=1).astype(np.float64))


def layout(z, kind, L):
    """Pencils of kind s as the input of the other kinds."""
    if kind == "s":
        return z
    if kind == "r":
        return np.stack([z.real, z.imag], axis=1)
    h = L // 2
    x = np.stack([z[:, :h + 1], np.roll(z, h, axis=1)[:, :h + 1]], axis=1).copy()
    x[:, :, [0, h]] = x[:, :, [0, h]].real
    return x


def made(L, rng):
    """One value throughout, square waves along every direction a step sums in,
    one value and two values alone, with components of equal size and mantissas
    just below two."""
    top = 2.0 - 2.0 ** -20
    n = np.arange(L)
    waves = [np.ones(L, complex)]
    for f in {1, 2, 3, L // 2, L // 3, L // 4, L // 5, L // 8, int(rng.integers(1, L))} - {0}:
        w = np.exp(2j * np.pi * f * (n + 0.25) / L)
        waves += [np.sign(w.real) + 1j * np.sign(w.imag), np.sign(w.real) * (1 + 1j), np.sign(w.real) * (1 - 1j)]
    for at in {0, 1, L // 3, L - 1}:
        one = np.zeros(L, complex)
        one[at] = 1 + 1j
        two = one.copy()
        two[(at + L // 2) % L] = 1 - 1j
        waves += [one, two]
    waves.append(rng.choice([-1.0, 1.0], L) + 1j * rng.choice([-1.0, 1.0], L))
    z = np.array(waves) + 0.0
    return np.concatenate([z * top, z * 1.5 * 2.0 ** 40, z * 1.01 * 2.0 ** -300])


def spectra(L, rng, power, count):
    k = np.maximum(np.minimum(np.arange(L), L - np.arange(L)), 1)
    return (rng.standard_normal((count, L)) + 1j * rng.standard_normal((count, L))) * k ** float(-power)


def test_made_pencils_stay_in_range(harness):
    exe, plans = harness
    assert len(plans) > 400
    for L, kind, radices in plans:
        x = layout(made(L, np.random.default_rng(L)), kind, L)
        err = rel(run(exe, L, kind, radices, x), transform(kind, wide(x), L))
        assert err.max() < 2.0 ** -52, (L, kind, radices, err.max(), int(err.argmax()))


@pytest.mark.parametrize("power", [0, 1, 2, 3, 4])
def test_no_less_precise_than_fp64(harness, power):
    exe, plans = harness
    for L, kind, radices in plans:
        if L < 32:  # few roundings: both are a unit of the result's last place
            continue
        x = layout(spectra(L, np.random.default_rng(7 * L + power), power, 12), kind, L)
        want = transform(kind, wide(x), L)
        ours, fp64 = rel(run(exe, L, kind, radices, x), want), rel(transform(kind, x, L), want)
        rms = [float(np.sqrt(np.mean(e ** 2))) for e in (ours, fp64)]
        assert rms[0] <= rms[1], (L, kind, radices, rms)


@pytest.mark.parametrize("L", [64, 72, 96, 100, 150, 288, 384, 432, 512, 576])
def test_errors_have_no_offset(harness, L):
    """The mean error of each output over many pencils is zero: the passes that
    follow sum an offset over the whole grid.  The mean of n errors exceeds t of
    their standard deviations with a probability below 2 exp(-n t^2 / 2); 0.1 at
    n = 4000 is 1e-4 for all outputs here together."""
    exe, plans = harness
    n = 4000
    for length, kind, radices in plans:
        if length != L:
            continue
        x = layout(spectra(L, np.random.default_rng(L), 0, n), kind, L)
        err = (run(exe, L, kind, radices, x) - transform(kind, wide(x), L)).astype(complex)
        sd = np.sqrt(np.mean(np.abs(err) ** 2, axis=0))
        off = np.abs(np.mean(err, axis=0)) / np.where(sd > 0, sd, 1)
        assert off.max() < 0.1, (kind, radices, off.max(), int(off.argmax()))
