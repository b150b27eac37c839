"""The work that users of this package have it do, as cases that can be timed.

Each case goes through the public Python binding (the same C ABI that a C++
host calls) and returns the particles, which is what the path computes:

* ``job``: one realisation, white noise to particles on the device
  (``Job.run``), in either arithmetic form, with NGenIC or MUSIC1 noise;
* ``batch``: an ensemble of uneven realisations as one captured graph;
* ``species``: a baryon + CDM run, both species assembled from one run's
  potentials, with masses;
* ``serve``: requests submitted to the server together, each result read and
  released.

``exact`` restates the whole path in plain torch and numpy in 64 bits.  It
shares with ``prepare`` only the inputs (seed, amplitude and PLT tables, growth
coefficients), not the computation.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from monofonic_gb300 import mfx

LATTICES = {"sc": mfx.SC, "bcc": mfx.BCC, "fcc": mfx.FCC}
SHIFTS = {"sc": [(0.0, 0.0, 0.0)],
          "bcc": [(0.0, 0.0, 0.0), (0.5, 0.5, 0.5)],
          "fcc": [(0.0, 0.0, 0.0), (0.0, 0.5, 0.5), (0.5, 0.0, 0.5), (0.5, 0.5, 0.0)]}
SECOND_SHIFT = {"sc": (0.5, 0.5, 0.5), "bcc": (0.5, 0.5, 0.0), "fcc": (0.5, 0.5, 0.5)}
OMEGA_M, OMEGA_B = 0.3, 0.045
DEVICE = "cuda:0"


def _job(name, n, box, z, order, lattice, form, noise="ngenic", fixing=False):
    return {"name": name, "kind": "job", "n": n, "box": box, "z": z, "order": order, "lattice": lattice,
            "plt": order == 3 and lattice != "sc", "form": form, "noise": noise, "fixing": fixing}


def listed():
    return [
        # a test run or a request of the smallest size: latency and launches
        _job("sc32_2lpt_fp32", 32, 250.0, 49.0, 2, "sc", "fp32c"),
        # the quick-start configuration: 64^3, the plain double-precision form
        _job("sc64_2lpt_fp64", 64, 100.0, 49.0, 2, "sc", "fp64"),
        # a grid that is no power of two, in double precision: padded length 150
        _job("bcc100_3lpt_fp64", 100, 150.0, 24.0, 3, "bcc", "fp64"),
        # the ordinary production box as the double-precision drop-in
        _job("bcc256_3lpt_fp64", 256, 300.0, 24.0, 3, "bcc", "fp64"),
        # the largest double-precision box that is run interactively
        _job("fcc384_3lpt_fp64", 384, 500.0, 24.0, 3, "fcc", "fp64"),
        # the same production box in the FP32-compensated form
        _job("bcc256_3lpt_fp32", 256, 300.0, 49.0, 3, "bcc", "fp32c"),
        # MUSIC1 white noise (filled Nyquist planes) in the FP32 form
        _job("bcc256_3lpt_music_fp32", 256, 300.0, 49.0, 3, "bcc", "fp32c", noise="music"),
        # a large box with PLT corrections, four particles a cell
        _job("fcc512_3lpt_fp32", 512, 1000.0 * 512 / 768, 24.0, 3, "fcc", "fp32c"),
        # the largest grid: 768^3 with fixed amplitudes (paired-and-fixed runs)
        _job("sc768_2lpt_fixed_fp32", 768, 1000.0, 24.0, 2, "sc", "fp32c", fixing=True),
        # an ensemble of uneven realisations in one captured graph
        {"name": "ensemble_fp32", "kind": "batch", "sizes": "128x8,192x6,256x2", "z": 49.0, "form": "fp32c"},
        # baryons and CDM from one set of potentials
        {"name": "species_bcc192_fp32", "kind": "species", "n": 192, "box": 300.0, "z": 49.0, "order": 3,
         "lattice": "bcc", "plt": True, "form": "fp32c"},
        # a burst of requests of mixed size, order and lattice
        {"name": "serve_mix_fp32", "kind": "serve", "form": "fp32c", "z": 49.0, "inflight": 2,
         "requests": "64:sc:1,128:bcc:3,96:fcc:2,192:sc:3,64:fcc:3,128:sc:2,192:bcc:2,64:bcc:2"},
    ]


def _log_size(rng, low, high, step):
    return max(low, min(high, int(math.exp(rng.uniform(math.log(low), math.log(high))) / step + 0.5) * step))


COMMON = [16, 32, 48, 64, 96, 128, 192, 256, 384, 512, 768]


def draw(rng):
    kind = rng.choice(["job"] * 8 + ["batch", "species", "serve"])
    if kind == "batch":
        return {"kind": "batch", "sizes": "%dx%d,%dx%d" % (rng.choice([32, 64, 96]), rng.randint(2, 10),
                                                           rng.choice([128, 192]), rng.randint(1, 8)),
                "z": float(rng.randint(49, 99)), "form": rng.choice(["fp32c", "fp32c", "fp64"])}
    lattice = rng.choice(["sc", "bcc", "fcc"])
    order = rng.choice([1, 2, 2, 3, 3])
    form = rng.choice(["fp64", "fp32c"])
    z = float(rng.randint(19, 63) if form == "fp64" else rng.randint(39, 99))
    if kind == "species":
        return {"kind": "species", "n": rng.choice([32, 64, 96, 128, 192]), "box": float(rng.randint(250, 600)), "z": z,
                "order": order, "lattice": lattice, "plt": lattice != "sc", "form": form}
    if kind == "serve":
        return {"kind": "serve", "form": form, "z": z, "inflight": 2,
                "requests": ",".join("%d:%s:%d" % (rng.choice([64, 96, 128]), rng.choice(["sc", "bcc", "fcc"]),
                                                   rng.randint(1, 3)) for _ in range(rng.randint(3, 8)))}
    top = (384 if lattice == "sc" else 256) if form == "fp64" else (512 if order == 3 or lattice != "sc" else 768)
    noise = rng.choice(["ngenic", "ngenic", "ngenic", "music"])
    if noise == "music":
        n = rng.choice([c for c in (32, 64, 128, 256) if c <= top])
    elif rng.random() < 0.3:
        n = _log_size(rng, 16, 256, 4)  # any admissible grid, padded lengths with other factors
    else:
        top_q = rng.uniform(math.log(16), math.log(top) + 0.2)
        n = min((c for c in COMMON if c <= top), key=lambda c: abs(math.log(c) - top_q))
    c = _job("", n, float(rng.randint(250, 1000)), z, order, lattice, form, noise, rng.random() < 0.3)
    del c["name"]
    c["plt"] = lattice != "sc" and rng.random() < 0.7
    return c


# ---------------------------------------------------------------------------
# inputs: what a user's program has before the call
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _engine():
    return mfx.Engine(0)


@functools.lru_cache(maxsize=None)
def _plt_table(lattice):
    return _engine().plt_table(LATTICES[lattice])


@functools.lru_cache(maxsize=16)
def _cosmology(n, box, z, order, lattice, sigma8):
    cosmo = mfx.Cosmology(mfx.ini_text(n, box, z, order, 1, lattice, sigma8=sigma8, omega_m=OMEGA_M,
                                       omega_b=OMEGA_B))
    coef = mfx.lpt_coefficients(cosmo.get("dplus_start"), cosmo.get("vfact_start"), order)
    return coef, cosmo.amp_table(n, box)


def _spec(seed, n, box, z, order, lattice, form, plt=False, noise="ngenic", fixing=False, sigma8=0.81):
    """The keyword arguments of one job (mfx.Job, mfx.Batch, mfx.Server)."""
    coef, amp = _cosmology(n, box, z, order, lattice, sigma8)
    spec = {"ngrid": n, "boxlen": box, "order": order, "amp_table": amp, "coef": coef, "lattice": LATTICES[lattice],
            "precision": mfx.FP64 if form == "fp64" else mfx.FP32C, "fixing": fixing, "lunit": box,
            "vunit": box / math.sqrt(1.0 / (1.0 + z)), "pos64": True, "vel64": form == "fp64", "id64": True,
            "plt_table": _plt_table(lattice) if plt else None}
    if noise == "music":
        spec.update(seed_table=None, noise_generator=mfx.NOISE_MUSIC1, music_seed=seed)
    else:
        spec.update(seed_table=mfx.ngenic_seed_table(seed, n))
    return spec


def _seed(seed, k=0):
    return 1 + (seed * 7919 + k * 104729) % 1_000_003


def _specs(case, seed):
    """The jobs of a case, in the order of its outputs, as (spec, lattice name)."""
    if case["kind"] == "batch":
        rng = np.random.RandomState(seed % (1 << 32))
        sizes = [int(n) for part in case["sizes"].split(",") for n, count in [part.split("x")] for _ in range(int(count))]
        return [(_spec(_seed(seed, k), n, float(rng.uniform(250.0, 500.0)), case["z"], 2, "sc", case["form"],
                       sigma8=float(rng.uniform(0.7, 0.9))), "sc") for k, n in enumerate(sizes)]
    if case["kind"] == "serve":
        asked = [r.split(":") for r in case["requests"].split(",")]
        return [(_spec(_seed(seed, k), int(n), 300.0, case["z"], int(order), lattice, case["form"],
                       plt=lattice != "sc"), lattice) for k, (n, lattice, order) in enumerate(asked)]
    return [(_spec(_seed(seed), case["n"], case["box"], case["z"], case["order"], case["lattice"], case["form"],
                   plt=case["plt"], noise=case.get("noise", "ngenic"), fixing=case.get("fixing", False)),
             case["lattice"])]


_tuned = set()


def _tune(spec):
    """The tile shapes of a size class, found once by a program that keeps its engine."""
    key = (spec["ngrid"], spec["order"], spec["precision"])
    if spec["precision"] == mfx.FP32C and key not in _tuned:
        job = mfx.Job(_engine(), **spec)
        job.autotune()
        job.close()
    _tuned.add(key)


class _Device:
    """Device memory that a job owns, for torch.as_tensor."""

    def __init__(self, address, shape, kind, owner):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": kind, "data": (address, False), "version": 3}
        self.owner = owner


def _views(job, seen):
    """The particle arrays of a job's last run as tensors of the job's own memory."""
    pos, vel, count = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_size_t()
    mfx.check(mfx.load().mfx_job_particles_device(job.handle, ctypes.byref(pos), ctypes.byref(vel), None,
                                                  ctypes.byref(count)))
    key = (pos.value, vel.value, count.value)
    if seen.get("key") != key:
        shape = (count.value, 3)
        seen["key"] = key
        seen["views"] = tuple(
            torch.as_tensor(_Device(p, shape, "<f8" if wide else "<f4", job), device=DEVICE)
            for p, wide in ((pos.value, job.pos64), (vel.value, job.vel64)))
    return seen["views"]


def _room(spec):
    """A user's own device arrays for one job's particles."""
    count = spec["ngrid"] ** 3 * (1 << spec["lattice"])
    return (torch.empty((count, 3), dtype=torch.float64, device=DEVICE),
            torch.empty((count, 3), dtype=torch.float64 if spec["vel64"] else torch.float32, device=DEVICE))


def prepare(case, seed):
    specs = _specs(case, seed)
    for spec, _ in specs:
        _tune(spec)
    only = specs[0][0]
    state = {"kind": case["kind"], "seen": [{} for _ in specs]}
    if case["kind"] == "batch":
        state["batch"] = mfx.Batch(_engine(), [spec for spec, _ in specs])
        state["jobs"] = [state["batch"].job(k) for k in range(len(specs))]
    elif case["kind"] == "serve":
        state["specs"] = [spec for spec, _ in specs]
        state["room"] = [_room(spec) for spec, _ in specs]
        state["server"] = mfx.Server(_engine(), case["inflight"])
    else:
        state["job"] = mfx.Job(_engine(), **only)
    if case["kind"] == "species":
        state["species"] = _species(case, only["amp_table"])
        state["room"] = [_room(only) + (torch.empty(only["ngrid"] ** 3 * (1 << only["lattice"]), dtype=torch.float64,
                                                    device=DEVICE),) for _ in state["species"]]
    return state


def _species(case, amp):
    """Baryon and CDM arguments with smooth density and velocity difference
    spectra of 5% and 1% of the matter amplitude."""
    kf = 2.0 * math.pi / case["box"]
    amplitude = amp * (kf * kf * np.arange(len(amp), dtype=np.float64))
    fb = OMEGA_B / OMEGA_M
    return [dict(secondary=sec, id_offset=off, c_species=c, mass_factor=om, amp_dbc=0.05 * amplitude,
                 amp_tbc=0.01 * amplitude)
            for sec, off, c, om in ((False, 0, -fb, OMEGA_M - OMEGA_B), (True, 1, 1.0 - fb, OMEGA_B))]


def run(state):
    kind = state["kind"]
    if kind == "job":
        state["job"].run()
        return _views(state["job"], state["seen"][0])
    if kind == "batch":
        state["batch"].run()
        state["batch"].wait()
        return [_views(job, seen) for job, seen in zip(state["jobs"], state["seen"])]
    if kind == "serve":
        server = state["server"]
        tickets = [server.submit(spec) for spec in state["specs"]]
        for ticket, (pos, vel) in zip(tickets, state["room"]):
            server.wait(ticket)
            server.job(ticket).fetch_particles_into(pos.data_ptr(), vel.data_ptr(), None)
            server.release(ticket)
        return state["room"]
    job = state["job"]
    job.run()
    for species, (pos, vel, mass) in zip(state["species"], state["room"]):
        job.set_species(**species)
        job.assemble(7)
        job.fetch_particles_into(pos.data_ptr(), vel.data_ptr(), None)
        mfx.check(mfx.load().mfx_job_fetch_masses(job.handle, ctypes.c_size_t(0), ctypes.c_size_t(job.num_particles),
                                                  ctypes.c_void_p(mass.data_ptr())))
    job.set_species(reset=True)
    return state["room"]


def _work_of(n, order, shifts, form, plt):
    """Tables read, particles written; the transforms of the dealiased products
    on the padded grid and of the six components of each sub-lattice."""
    real = 8 if form == "fp64" else 4
    particles = shifts * n ** 3
    size = 4 * n * n + 8 * (3 * (n // 2) ** 2 + 1) + (4 * 64 * 64 * 33 * 8 if plt else 0)
    size += particles * (24 + 3 * real)
    m = 3 * n // 2
    transforms = {1: 0, 2: 7, 3: 27}[order]
    flops = 2.5 * transforms * m ** 3 * math.log2(m ** 3) + 2.5 * 6 * shifts * n ** 3 * math.log2(n ** 3)
    return size, flops


def work(case):
    if case["kind"] == "batch":
        parts = [_work_of(int(n), 2, 1, case["form"], False) for part in case["sizes"].split(",")
                 for n, count in [part.split("x")] for _ in range(int(count))]
    elif case["kind"] == "serve":
        parts = [_work_of(int(n), int(order), len(SHIFTS[lattice]), case["form"], lattice != "sc")
                 for n, lattice, order in (r.split(":") for r in case["requests"].split(","))]
    else:
        parts = [_work_of(case["n"], case["order"], len(SHIFTS[case["lattice"]]), case["form"], case["plt"])]
        if case["kind"] == "species":
            n, shifts = case["n"], len(SHIFTS[case["lattice"]])
            second = 2.5 * 8 * shifts * n ** 3 * math.log2(n ** 3)
            parts.append((shifts * n ** 3 * (24 + (24 if case["form"] == "fp64" else 12) + 16), second))
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


# ---------------------------------------------------------------------------
# the same path in 64 bits, in plain torch and numpy
# ---------------------------------------------------------------------------
def _ranlux_words(seeds, count):
    """The first `count` 48-bit words of RANLUX (luxury 1 of the double-precision
    variant) for each seed: [count][column]."""
    reg = seeds.to(torch.int64).clone()
    reg[reg == 0] = 1
    bits = [(reg >> q) & 1 for q in range(31)]
    ib, jb = 0, 18
    y = []
    for _ in range(12):
        word = torch.zeros_like(reg)
        for _ in range(48):
            word = 2 * word + (1 - bits[ib])
            bits[ib] = bits[ib] ^ bits[jb]
            ib, jb = (ib + 1) % 31, (jb + 1) % 31
        y.append(word)
    mask = (1 << 48) - 1
    borrow = torch.zeros_like(reg)  # 0 or -1
    out = torch.empty((count, reg.numel()), dtype=torch.int64, device=reg.device)
    made = 0
    while made < count:
        for t in range(202):
            d = y[7] - y[0]
            d += borrow
            borrow = d >> 63
            d &= mask
            y = y[1:] + [d]
        for d in y[:count - made]:
            out[made] = d
            made += 1
    return out


def _ngenic_noise(table, n):
    """White noise in k-space, one generator stream per column, Hermitian on kz = 0."""
    h = n // 2
    words = _ranlux_words(torch.from_numpy(np.asarray(table, dtype=np.int64)).to(DEVICE), 2 * h)
    words = words.reshape(h, 2, n, n)
    w = torch.zeros((n, n, h + 1), dtype=torch.complex128, device=DEVICE)
    for k in range(h):
        u = words[k].to(torch.float64) * 2.0 ** -48
        w[:, :, k] = torch.polar(torch.sqrt(-torch.log(u[1])), u[0] * (2.0 * math.pi))
    del words
    w[h] = 0.0
    w[:, h] = 0.0
    p = w[:, :, 0].clone()
    back = (-torch.arange(n, device=DEVICE)) % n
    keep = torch.zeros((n, n), dtype=torch.bool, device=DEVICE)
    keep[1:h] = True
    keep[0, 1:h] = True
    keep[:, h] = False
    p = torch.where(keep, p, torch.zeros_like(p))
    w[:, :, 0] = p + p[back][:, back].conj()
    return w


def _music_noise(seed, n, cube=32):
    """White noise in real space, one Mersenne Twister per cube and the ratio of
    uniforms method, transformed (its mean lies at k = 0, which is not used)."""
    cs = min(cube, n)
    nc = n // cs
    out = np.empty((n, n, n))
    for c in range(nc ** 3):
        rng = np.random.RandomState(seed + c)
        got, need = [], cs ** 3
        while need > 0:
            pairs = int(1.45 * need) + 64
            x = np.frombuffer(rng.bytes(8 * pairs), dtype="<u4").astype(np.float64) / 4294967296.0
            u = 1.0 - x[0::2]
            v = (x[1::2] - 0.5) * 1.7156
            a, b = u - 0.449871, np.abs(v) + 0.386595
            q = a * a + b * (0.19600 * b - 0.25472 * a)
            ok = (q < 0.27597) | ((q <= 0.27846) & (v * v <= -4.0 * u * u * np.log(u)))
            got.append((v[ok] / u[ok])[:need])
            need -= len(got[-1])
        i, j, k = c // (nc * nc), c // nc % nc, c % nc
        out[i * cs:(i + 1) * cs, j * cs:(j + 1) * cs, k * cs:(k + 1) * cs] = np.concatenate(got).reshape(cs, cs, cs)
    return torch.fft.rfftn(torch.from_numpy(out).to(DEVICE), norm="ortho")


def _planes(c, n):
    """The Hermitian part of the kz = 0 and kz = n/2 planes, which is what a
    real transform along z, taken last, makes of them."""
    back = (-torch.arange(n, device=DEVICE)) % n
    for kz in (0, c.shape[2] - 1):
        p = c[:, :, kz]
        c[:, :, kz] = 0.5 * (p + p[back][:, back].conj())
    return c


def _to_real(c, n):
    return torch.fft.irfftn(_planes(c, n), s=(n, n, n), norm="ortho")


def _index(n, count):
    i = torch.arange(count, dtype=torch.float64, device=DEVICE)
    return torch.where(i > n // 2, i - n, i)


class _Grid:
    """Derivatives, dealiased products and sub-lattice shifts on one grid."""

    def __init__(self, n, box):
        self.n, self.m, self.box = n, 3 * n // 2, box
        kf = 2.0 * math.pi / box
        self.k = [(_index(n, c) * kf).reshape(s) for c, s in ((n, (n, 1, 1)), (n, (1, n, 1)),
                                                              (n // 2 + 1, (1, 1, n // 2 + 1)))]
        self.g = []
        for k in self.k:
            g = k.clone().reshape(-1)
            g[n // 2] = 0.0
            self.g.append(g.reshape(k.shape))
        self.k2 = self.k[0] ** 2 + self.k[1] ** 2 + self.k[2] ** 2
        i = torch.arange(n, device=DEVICE)
        self.at = torch.where(i > n // 2, i + n // 2, i)

    def hessian(self, f, a, b):
        """-k_a k_b f on the padded real grid."""
        m, n = self.m, self.n
        big = torch.zeros((m, m, m // 2 + 1), dtype=torch.complex128, device=DEVICE)
        return self._pad(f * (-(self.g[a] * self.g[b])), big, m, n)

    def padded(self, f):
        m, n = self.m, self.n
        return self._pad(f, torch.zeros((m, m, m // 2 + 1), dtype=torch.complex128, device=DEVICE), m, n)

    def _pad(self, f, big, m, n):
        big[self.at[:, None], self.at[None, :], :n // 2 + 1] = f * 1.5 ** 1.5
        return _to_real(big, m)

    def unpad(self, r):
        n, h = self.n, self.n // 2
        big = torch.fft.rfftn(r, norm="ortho")
        out = big[:, :, :h + 1][self.at][:, self.at] / 1.5 ** 1.5
        out[h], out[:, h], out[:, :, h] = 0.0, 0.0, 0.0
        return out

    def inverse_laplacian(self, f):
        out = -f / self.k2
        out[0, 0, 0] = 0.0
        return out

    def shift(self, r, s):
        c = torch.fft.rfftn(r, norm="ortho")
        dx = self.box / self.n
        for axis in range(3):
            if s[axis]:
                c = c * torch.polar(torch.ones_like(self.k[axis]), self.k[axis] * (s[axis] * dx))
        return _to_real(c, self.n)


def _potentials(grid, phi, order):
    phi2 = phi3 = None
    a3 = []
    if order > 1:
        pairs = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
        h = {p: grid.hessian(phi, *p) for p in pairs}
        src = h[0, 0] * (h[1, 1] + h[2, 2]) + h[1, 1] * h[2, 2]
        for p in pairs[3:]:
            src -= h[p] * h[p]
        phi2 = grid.inverse_laplacian(grid.unpad(src))
        del src
    if order > 2:
        total = None
        for fac, a, b, c in ((1.0, (0, 0), (1, 1), (2, 2)), (2.0, (0, 1), (0, 2), (1, 2)),
                             (-1.0, (1, 2), (1, 2), (0, 0)), (-1.0, (0, 2), (0, 2), (1, 1)),
                             (-1.0, (0, 1), (0, 1), (2, 2))):
            t = grid.padded(grid.unpad(h[a] * h[b])) * h[c] * fac
            total = t if total is None else total.add_(t)
        g = {p: grid.hessian(phi2, *p) for p in pairs}
        for a, b, c in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
            total -= 5.0 / 7.0 * h[a, a] * (g[b, b] + g[c, c])
        for p in pairs[3:]:
            total += 10.0 / 7.0 * h[p] * g[p]
        phi3 = grid.inverse_laplacian(grid.unpad(total))
        del total

        def at(x, i, j):
            return x[min(i, j), max(i, j)]

        for d in range(3):
            e, f = (d + 1) % 3, (d + 2) % 3
            t = at(g, d, e) * at(h, d, f) - at(g, d, f) * at(h, d, e)
            t += at(h, e, f) * (at(g, e, e) - at(g, f, f))
            t -= at(g, e, f) * (at(h, e, e) - at(h, f, f))
            a3.append(grid.inverse_laplacian(grid.unpad(t)))
    return phi2, phi3, a3


def _cic(table, x, y, z):
    """Trilinear interpolation in the 64 x 64 x 33 tables (periodic in x and y)."""
    at = [torch.floor(v).to(torch.int64) for v in (x, y, z)]
    d = [v - i for v, i in zip((x, y, z), at)]
    nxt = [(at[0] + 1) % 64, (at[1] + 1) % 64, torch.clamp(at[2] + 1, max=32)]
    out = 0.0
    for a in (0, 1):
        for b in (0, 1):
            for c in (0, 1):
                i, j, k = (nxt[0] if a else at[0]), (nxt[1] if b else at[1]), (nxt[2] if c else at[2])
                w = (d[0] if a else 1.0 - d[0])[:, None, None] * (d[1] if b else 1.0 - d[1])[None, :, None]
                w = w * (d[2] if c else 1.0 - d[2])[None, None, :]
                out = out + table[i[:, None, None], j[None, :, None], k[None, None, :]] * w
    return out


def _gradient(n, box, table):
    """The gradient's imaginary factors and the velocity correction: i k, or the
    eigenmodes of the particle lattice."""
    grid = _Grid(n, box)
    if table is None:
        return grid.g, 1.0
    t = torch.from_numpy(np.asarray(table)).to(DEVICE)
    ratio = 64.0 / n
    at = [torch.arange(c, dtype=torch.float64, device=DEVICE) * ratio for c in (n, n, n // 2 + 1)]
    k = [((v - (v > 32.0) * 64.0) * (2.0 * math.pi)).reshape(s) for v, s in zip(at, ((n, 1, 1), (1, n, 1),
                                                                                     (1, 1, n // 2 + 1)))]
    kr = torch.sqrt(k[0] ** 2 + k[1] ** 2 + k[2] ** 2)
    one = torch.where(kr > 0, kr, torch.ones_like(kr))
    ct = torch.where(kr > 0, k[2] / one, torch.ones_like(kr))
    kp = torch.sqrt(k[0] ** 2 + k[1] ** 2) + 0.0 * k[2]
    st = torch.where(kr > 0, kp / one, torch.zeros_like(kr))
    onep = torch.where(kp > 0, kp, torch.ones_like(kp))
    cp = torch.where(kp > 0, k[0] / onep, torch.ones_like(kp))
    sp = torch.where(kp > 0, k[1] / onep, torch.zeros_like(kp))
    del one, onep, kp
    kmod = kr / ratio / box
    dr, dt, dp, vc = (_cic(t[q], *at) for q in range(4))
    return [kmod * (dr * st * cp + dt * ct * cp - dp * sp), kmod * (dr * st * sp + dt * ct * sp + dp * cp),
            kmod * (dr * ct - dt * st)], vc


def _exact_job(spec, lattice, species=(None,)):
    """[(positions, velocities[, masses])] of one job, per species."""
    n, box, order, coef = spec["ngrid"], spec["boxlen"], spec["order"], spec["coef"]
    w = (_ngenic_noise(spec["seed_table"], n) if spec["seed_table"] is not None
         else _music_noise(spec["music_seed"], n))
    if spec["fixing"]:
        size = w.abs()
        w = torch.where(size > 0, w / torch.where(size > 0, size, torch.ones_like(size)), w)
        del size
    w /= (box / n / 2.0 / math.pi) ** 1.5
    grid = _Grid(n, box)
    i = [_index(n, c) ** 2 for c in (n, n, n // 2 + 1)]
    square = (i[0][:, None, None] + i[1][None, :, None] + i[2][None, None, :]).to(torch.int64)

    def per_mode(table):
        return torch.from_numpy(np.asarray(table, dtype=np.float64)).to(DEVICE)[square]

    phi = -w * per_mode(spec["amp_table"])
    phi[0, 0, 0] = 0.0
    w[0, 0, 0] = 0.0
    phi2, phi3, a3 = _potentials(grid, phi, order)
    grad, vc = _gradient(n, box, spec["plt_table"])
    total = phi * coef["g1"]
    moving = phi * (coef["g1"] * coef["vfac1"])
    if order > 1:
        phi2 *= coef["g2"]
        total += phi2
        moving += coef["vfac2"] * phi2
    if order > 2:
        phi3 *= coef["g3"]
        total += phi3
        moving += coef["vfac3"] * phi3
        a3 = [a * coef["g3c"] for a in a3]
    del phi, phi2, phi3
    shifts = SHIFTS[lattice]
    cells = n ** 3
    count = len(shifts) * cells
    made = []
    for sp in species:
        second = SECOND_SHIFT[lattice] if sp and sp["secondary"] else (0.0, 0.0, 0.0)

        def read_out(c, out, offset=None):
            r = _to_real(c, n) if c.is_complex() else c
            if any(second):
                r = grid.shift(r, second)
            for q, s in enumerate(shifts):
                if q > 0:
                    r = grid.shift(r, tuple(a - b for a, b in zip(s, shifts[q - 1])))
                out[q * cells:(q + 1) * cells] = (r if offset is None else r + offset(s)).reshape(-1)

        pos = torch.empty((count, 3), dtype=torch.float64, device=DEVICE)
        vel = torch.empty((count, 3), dtype=torch.float64, device=DEVICE)
        for d in range(3):
            e, f = (d + 1) % 3, (d + 2) % 3
            curl = grad[e] * a3[f] - grad[f] * a3[e] if order > 2 else 0.0
            c = (grad[d] * total + curl) * (1j * spec["lunit"] / box)
            c[0, 0, 0] = 0.0
            shape = [1, 1, 1]
            shape[d] = n
            lattice_at = torch.arange(n, dtype=torch.float64, device=DEVICE).reshape(shape)
            read_out(c, pos[:, d], lambda s: (lattice_at + (s[d] + second[d])) / n * spec["lunit"])
            c = (grad[d] * moving + (coef["vfac3"] * curl if order > 2 else 0.0)) * 1j
            if sp:
                t = w * per_mode(sp["amp_tbc"]) * (1j * coef["vfac1"] * sp["c_species"]) * grad[d] / grid.k2
                t[0, 0, 0] = 0.0
                c -= t
            c *= vc * (spec["vunit"] / box)
            c[0, 0, 0] = 0.0
            read_out(c, vel[:, d])
        out = (pos, vel)
        if sp:
            mass = torch.empty(count, dtype=torch.float64, device=DEVICE)
            rho = _to_real(w * per_mode(sp["amp_dbc"]), n)
            read_out((1.0 + sp["c_species"] * rho) * sp["mass_factor"], mass)
            out = (pos, vel, mass / count)
        made.append(out)
    return made


def exact(case, seed):
    specs = _specs(case, seed)
    if case["kind"] == "job":
        return _exact_job(*specs[0])[0]
    if case["kind"] == "species":
        spec, lattice = specs[0]
        return _exact_job(spec, lattice, _species(case, spec["amp_table"]))
    return [_exact_job(spec, lattice)[0] for spec, lattice in specs]
