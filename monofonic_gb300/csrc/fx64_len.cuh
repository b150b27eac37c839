// The fixed-point transforms (fx64.cuh) compiled for one length: the kernels
// of fx64.cu with radices, index arithmetic and thread counts folded to
// constants, the first step of an x or y pass reading HBM straight into
// registers and the last one writing from them (one shared-memory exchange for
// two steps).  Lengths without an instance take the run-time kernels.
#pragma once
#include "fx64.cuh"
#include "fx64.h"

namespace fx {

__device__ __forceinline__ int dbl_exponent(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }
__device__ __forceinline__ double nan_of() { return __longlong_as_double(0x7ff8000000000000LL); }

// radices of a length (the smallest, whose butterflies carry no twiddles, first)
// and threads per CTA of eight pencils
template <int L> struct Len;
#define FX_LEN(L_, STEPS_, A_, B_, C_, T_)                                    \
  template <> struct Len<L_> {                                               \
    static constexpr int steps = STEPS_, T = T_;                              \
    static FX_HD constexpr int R(int q) { return q == 0 ? A_ : (q == 1 ? B_ : C_); } \
  };
FX_LEN(16, 2, 4, 4, 1, 32)
FX_LEN(24, 2, 4, 6, 1, 64)
FX_LEN(32, 2, 4, 8, 1, 64)
FX_LEN(48, 2, 6, 8, 1, 64)
FX_LEN(64, 2, 8, 8, 1, 64)
FX_LEN(72, 2, 8, 9, 1, 96)
FX_LEN(96, 2, 8, 12, 1, 96)
FX_LEN(128, 2, 8, 16, 1, 128)
FX_LEN(144, 2, 12, 12, 1, 96)
FX_LEN(192, 2, 12, 16, 1, 128)
FX_LEN(256, 2, 16, 16, 1, 128)
FX_LEN(288, 2, 16, 18, 1, 160)
FX_LEN(384, 2, 16, 24, 1, 192)
FX_LEN(512, 3, 8, 8, 8, 256)
FX_LEN(576, 2, 24, 24, 1, 192)
FX_LEN(768, 3, 8, 8, 12, 256)
FX_LEN(1152, 3, 8, 12, 12, 384)
#undef FX_LEN

// resident CTAs that the register file is shared by at `regs` registers a thread
#ifndef FX_REG_S
#define FX_REG_S 168
#endif
#ifndef FX_REG_Z
#define FX_REG_Z 112
#endif
constexpr int min_ctas(int T, int regs) { return 65536 / (T * regs) > 0 ? 65536 / (T * regs) : 1; }

template <int L> struct Fft {
  using D = Len<L>;
  static constexpr int P = 8, lgP = 3, T = D::T, steps = D::steps, items_max = P * L;
  static FX_HD constexpr int NS(int q) { return q == 0 ? 1 : NS(q - 1) * D::R(q - 1); }
  // butterflies of step q a thread holds
  static FX_HD constexpr int MU(int q) { return (P * (L / D::R(q)) + T - 1) / T; }
  static constexpr int smem = L * P * 16 + P * 8;

  static __device__ __forceinline__ int slot(int e, int pen) { return (e << lgP) + (pen ^ (e & (P - 1))); }

  // registers of one step
  template <int Q> struct Regs {
    I2 v[MU(Q)][D::R(Q)];
  };
  template <int Q> static __device__ __forceinline__ bool live(int m) {
    constexpr int items = P * (L / D::R(Q));
    return items % T == 0 || int(threadIdx.x) + m * T < items;
  }
  template <int Q> static __device__ __forceinline__ int jof(int m) { return (int(threadIdx.x) + m * T) >> lgP; }
  // element index of input r / output r of butterfly j
  template <int Q> static __device__ __forceinline__ int in_of(int j, int r) { return j + r * (L / D::R(Q)); }
  template <int Q> static __device__ __forceinline__ int out_of(int j, int r) {
    constexpr int ns = NS(Q), R = D::R(Q);
    return (j / ns) * (ns * R) + j % ns + r * ns;
  }
  template <int Q> static __device__ __forceinline__ void load(Regs<Q> &g, const longlong2 *s, int pen) {
#pragma unroll
    for (int m = 0; m < MU(Q); ++m)
      if (live<Q>(m)) {
        const int j = jof<Q>(m);
#pragma unroll
        for (int r = 0; r < D::R(Q); ++r) {
          const longlong2 w = s[slot(in_of<Q>(j, r), pen)];
          g.v[m][r] = {w.x, w.y};
        }
      }
  }
  template <int Q> static __device__ __forceinline__ void store(const Regs<Q> &g, longlong2 *s, int pen) {
#pragma unroll
    for (int m = 0; m < MU(Q); ++m)
      if (live<Q>(m)) {
        const int j = jof<Q>(m);
#pragma unroll
        for (int r = 0; r < D::R(Q); ++r) s[slot(out_of<Q>(j, r), pen)] = make_longlong2(g.v[m][r].x, g.v[m][r].y);
      }
  }
  template <int Q> static __device__ __forceinline__ void butterfly(Regs<Q> &g, const longlong2 *tw) {
    constexpr int R = D::R(Q), ns = NS(Q);
#pragma unroll
    for (int m = 0; m < MU(Q); ++m)
      if (live<Q>(m)) {
        if constexpr (Q > 0) {
          const longlong2 *w = tw;
          const int inc = (jof<Q>(m) % ns) * (L / (ns * R));
          g.v[m][0] = eighth(g.v[m][0]);
#pragma unroll
          for (int r = 1; r < R; ++r) g.v[m][r] = twiddle8(g.v[m][r], __ldg(&w[r * inc]));
        }
        Dft<R>::run(g.v[m]);
      }
  }
  // steps Q0 .. last, the last one's outputs left in registers
  template <int Q0, class F> static __device__ __forceinline__ void rest(longlong2 *s, int pen, const longlong2 *tw,
                                                                        F &&out) {
    Regs<Q0> g;
    load<Q0>(g, s, pen);
    butterfly<Q0>(g, tw);
    if constexpr (Q0 + 1 < steps) {
      __syncthreads();
      store<Q0>(g, s, pen);
      __syncthreads();
      rest<Q0 + 1>(s, pen, tw, out);
    } else {
      out(g);
    }
  }
  static constexpr int last = D::steps - 1;
};

struct LArgs {
  const longlong2 *tw;
  int B;
  Strided s;
};
struct LRows {
  const longlong2 *tw;
  int B;
  Rows r;
};

template <int L, bool TRUNC> __global__ void __launch_bounds__(Len<L>::T, min_ctas(Len<L>::T, FX_REG_S)) k_fx_strided_l(const __grid_constant__ LArgs a) {
  using F = Fft<L>;
  extern __shared__ __align__(16) longlong2 sm[];
  const Strided &d = a.s;
  const int t = threadIdx.x, pen = t & 7;
  int *emax = reinterpret_cast<int *>(sm + L * F::P);
  const int kblocks = (d.kc + 7) >> 3;
  const int o = blockIdx.x / kblocks, kz0 = (blockIdx.x - o * kblocks) << 3, kz = kz0 + pen;
  const bool lv = kz < d.kc;
  const int n = d.n, nh = n >> 1;
  for (int op = d.first[blockIdx.y]; op < d.first[blockIdx.y + 1]; ++op) {
    if (t < 8) emax[t] = 0;
    const double2 *src = d.src[op] + (long long)o * d.in_outer + kz;
    const int pr = d.pr[op], pk = d.pk[op];
    typename F::template Regs<0> g;
    int em = 0;
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
        const int j = F::template jof<0>(m);
#pragma unroll
        for (int r = 0; r < F::D::R(0); ++r) {
          const int l = F::template in_of<0>(j, r);
          const int i = !d.pad_in ? l : (l <= nh ? l : (l > n ? l - nh : -1));
          double2 v = make_double2(0.0, 0.0);
          if (lv && i >= 0) v = src[(long long)i * d.in_row];
          g.v[m][r] = {__double_as_longlong(v.x), __double_as_longlong(v.y)};
        }
      }
    if ((pr | pk) != 0) {
      const double kf = pk == 0 ? 1.0 : (kz == nh ? 0.0 : (pk == 1 ? double(kz) : double(kz) * double(kz)));
#pragma unroll
      for (int m = 0; m < F::MU(0); ++m)
        if (F::template live<0>(m)) {
          const int j = F::template jof<0>(m);
#pragma unroll
          for (int r = 0; r < F::D::R(0); ++r) {
            const int l = F::template in_of<0>(j, r);
            const int i = !d.pad_in ? l : (l <= nh ? l : (l > n ? l - nh : -1));
            if (i >= 0) {
              const double f = (pr ? __ldg(&d.mode[(pr - 1) * n + i]) : 1.0) * kf;
              g.v[m][r].x = __double_as_longlong(__longlong_as_double(g.v[m][r].x) * f);
              g.v[m][r].y = __double_as_longlong(__longlong_as_double(g.v[m][r].y) * f);
            }
          }
        }
    }
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
#pragma unroll
        for (int r = 0; r < F::D::R(0); ++r)
          em = max(em, max(dbl_exponent(__longlong_as_double(g.v[m][r].x)), dbl_exponent(__longlong_as_double(g.v[m][r].y))));
      }
    em = max(em, __shfl_xor_sync(0xffffffffu, em, 8));
    em = max(em, __shfl_xor_sync(0xffffffffu, em, 16));
    __syncthreads();
    if ((t & 31) < 8) atomicMax(&emax[pen], em);
    __syncthreads();
    em = emax[pen];
    const bool bad = em == 2047;
    int S = em - 1022 - a.B + 3 * (F::steps - 1);
    const bool inv = d.inverse;
    const int sh = em + 63 - a.B;
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
#pragma unroll
        for (int r = 0; r < F::D::R(0); ++r) {
          const double x = __longlong_as_double(g.v[m][r].x), y = __longlong_as_double(g.v[m][r].y);
          g.v[m][r] = {to_fixed(inv ? y : x, sh), to_fixed(inv ? x : y, sh)};
        }
      }
    F::template butterfly<0>(g, a.tw);
    F::template store<0>(g, sm, pen);
    __syncthreads();
    auto put = [&](auto &h) {
      double2 *dst = d.dst[op] + (long long)o * d.out_outer + kz;
      const int so = o > nh ? o - n : o;
      const bool swap = TRUNC || inv;
#pragma unroll
      for (int m = 0; m < F::MU(F::last); ++m)
        if (F::template live<F::last>(m)) {
          const int j = F::template jof<F::last>(m);
#pragma unroll
          for (int r = 0; r < F::D::R(F::last); ++r) {
            const int l = F::template out_of<F::last>(j, r);
            const int i = !d.cut_out ? l : (l <= nh ? l : (l > n ? l - nh : -1));
            if (i >= 0 && lv) {
              double2 v = make_double2(to_double(swap ? h.v[m][r].y : h.v[m][r].x, S),
                                       to_double(swap ? h.v[m][r].x : h.v[m][r].y, S));
              if (bad) v = make_double2(nan_of(), nan_of());
              if (TRUNC) {
                v.x *= d.fac;
                v.y *= d.fac;
              } else if (d.cut_out) {
                if (i == nh || (d.inv_lap && (o == nh || (o | i | kz) == 0))) {
                  v = make_double2(0.0, 0.0);
                } else if (d.inv_lap) {
                  const int si = i > nh ? i - n : i;
                  const double f = -d.fac * __ldg(&d.rinv[so * so + si * si + kz * kz]);
                  v.x *= f;
                  v.y *= f;
                }
              }
              dst[(long long)i * d.out_row] = v;
            }
          }
        }
    };
    if constexpr (!TRUNC) {
      F::template rest<1>(sm, pen, a.tw, put);
    } else {
      // forward transform, the N-grid modes kept, the largest brought back
      // below 2^B, transformed back (inverse = exchange, forward, exchange)
      if (t < 8) emax[t] = 0;
      int bits = 0;
      F::template rest<1>(sm, pen, a.tw, [&](auto &h) {
#pragma unroll
        for (int m = 0; m < F::MU(F::last); ++m)
          if (F::template live<F::last>(m)) {
            const int j = F::template jof<F::last>(m);
#pragma unroll
            for (int r = 0; r < F::D::R(F::last); ++r) {
              const int l = F::template out_of<F::last>(j, r);
              const bool keep = l < nh || l > n;
              const I2 v = h.v[m][r];
              h.v[m][r] = keep ? I2{v.y, v.x} : I2{0, 0};
              if (keep) bits = max(bits, 64 - min(__clzll(v.x ^ (v.x >> 63)), __clzll(v.y ^ (v.y >> 63))));
            }
          }
        bits = max(bits, __shfl_xor_sync(0xffffffffu, bits, 8));
        bits = max(bits, __shfl_xor_sync(0xffffffffu, bits, 16));
        __syncthreads();
        if ((t & 31) < 8) atomicMax(&emax[pen], bits);
        F::template store<F::last>(h, sm, pen);
        __syncthreads();
      });
      const int down = emax[pen] - a.B;
      const int dn = max(down, 0), up = max(-down, 0);
      const long long half = dn ? 1LL << (dn - 1) : 0;
      F::template load<0>(g, sm, pen);
#pragma unroll
      for (int m = 0; m < F::MU(0); ++m)
        if (F::template live<0>(m)) {
#pragma unroll
          for (int r = 0; r < F::D::R(0); ++r)
            g.v[m][r] = {((g.v[m][r].x + half) >> dn) << up, ((g.v[m][r].y + half) >> dn) << up};
        }
      S += down + 3 * (F::steps - 1);
      F::template butterfly<0>(g, a.tw);
      __syncthreads();
      F::template store<0>(g, sm, pen);
      __syncthreads();
      F::template rest<1>(sm, pen, a.tw, put);
    }
    if (!TRUNC && d.inv_lap && kz0 + 8 >= d.kc) {
      double2 *z = d.dst[op] + (long long)o * d.out_outer + d.kc;  // the kz Nyquist column
      for (int i = t; i < n; i += F::T) z[(long long)i * d.out_row] = make_double2(0.0, 0.0);
    }
    __syncthreads();
  }
}

// spectra -> real rows (fx64.cu k_fx_c2r)
template <int L> __global__ void __launch_bounds__(Len<L>::T, min_ctas(Len<L>::T, FX_REG_Z)) k_fx_c2r_l(const __grid_constant__ LRows a) {
  using F = Fft<L>;
  extern __shared__ __align__(16) longlong2 sm[];
  const Rows &d = a.r;
  constexpr int h = L / 2, W = F::T / 32;
  const int t = threadIdx.x, lane = t & 31, pen = t & 7;
  int *emax = reinterpret_cast<int *>(sm + L * F::P);
  double *base = d.field[blockIdx.y];
  const long long row0 = (long long)blockIdx.x * 16;
  const int kc = min(d.kc, h);
  const bool nyq = d.kc > h;
  if (t < 8) emax[t] = 0;
  for (int e = t; e < (L - 2 * kc + 1) * 8; e += F::T) sm[F::slot(kc + (e >> 3), e & 7)] = make_longlong2(0, 0);
  __syncthreads();
  for (int q = t >> 5; q < 16; q += W) {
    const long long row = row0 + q;
    const bool lv = row < d.rows;
    const double2 *src = reinterpret_cast<const double2 *>(base + row * d.pitch);
    const int p = q >> 1, second = q & 1;
    int em = 0;
    constexpr int NL = (h + 31) / 32;
    double2 v[NL];
#pragma unroll
    for (int c = 0; c < NL; ++c) {
      const int k = lane + 32 * c;
      v[c] = make_double2(0.0, 0.0);
      if (lv && k < kc) v[c] = src[k];
    }
#pragma unroll
    for (int c = 0; c < NL; ++c) {
      const int k = lane + 32 * c;
      if (k >= kc) continue;
      if (k == 0) {
        em = max(em, dbl_exponent(v[c].x));
        reinterpret_cast<double *>(&sm[F::slot(0, p)])[second] = v[c].x;
      } else {
        em = max(em, max(dbl_exponent(v[c].x), dbl_exponent(v[c].y)));
        sm[F::slot(second ? L - k : k, p)] = make_longlong2(__double_as_longlong(v[c].x), __double_as_longlong(v[c].y));
      }
    }
    if (nyq && lane == 0) {
      const double x = lv ? src[h].x : 0.0;
      em = max(em, dbl_exponent(x));
      reinterpret_cast<double *>(&sm[F::slot(h, p)])[second] = x;
    }
    em = int(__reduce_max_sync(0xffffffffu, unsigned(em)));
    if (lane == 0) atomicMax(&emax[p], em);
  }
  __syncthreads();
  {
    const int sh = emax[pen] + 63 - a.B;
    for (int k = t >> 3; k < kc; k += F::T / 8) {
      longlong2 &wa = sm[F::slot(k, pen)];
      const longlong2 va = wa;
      const long long ax = to_fixed(__longlong_as_double(va.x), sh), ay = to_fixed(__longlong_as_double(va.y), sh);
      if (k == 0) {
        wa = make_longlong2(ay, ax);
        continue;
      }
      longlong2 &wb = sm[F::slot(L - k, pen)];
      const longlong2 vb = wb;
      const long long bx = to_fixed(__longlong_as_double(vb.x), sh), by = to_fixed(__longlong_as_double(vb.y), sh);
      wa = make_longlong2(ay + bx, ax - by);
      wb = make_longlong2(bx - ay, ax + by);
    }
    if (nyq && t < 8) {
      longlong2 &w = sm[F::slot(h, t)];
      const longlong2 v = w;
      w = make_longlong2(to_fixed(__longlong_as_double(v.y), sh), to_fixed(__longlong_as_double(v.x), sh));
    }
  }
  __syncthreads();
  F::template rest<0>(sm, pen, a.tw, [&](auto &g) {
    __syncthreads();
    F::template store<F::last>(g, sm, pen);
    __syncthreads();
  });
  for (int q = t >> 5; q < 16; q += W) {
    const long long row = row0 + q;
    if (row >= d.rows) break;
    double *dst = base + row * d.pitch;
    const int p = q >> 1, second = q & 1;
    const int S = emax[p] - 1022 - a.B + 3 * (F::steps - 1);
    const bool bad = emax[p] == 2047;
#pragma unroll 4
    for (int e = lane; e < L; e += 32) {
      const long long v = reinterpret_cast<const long long *>(&sm[F::slot(e, p)])[1 - second];
      dst[e] = bad ? nan_of() : to_double(v, S);
    }
  }
}

// real rows -> spectra (fx64.cu k_fx_r2c)
template <int L> __global__ void __launch_bounds__(Len<L>::T, min_ctas(Len<L>::T, FX_REG_Z)) k_fx_r2c_l(const __grid_constant__ LRows a) {
  using F = Fft<L>;
  extern __shared__ __align__(16) longlong2 sm[];
  const Rows &d = a.r;
  constexpr int W = F::T / 32;
  const int t = threadIdx.x, lane = t & 31, pen = t & 7;
  int *emax = reinterpret_cast<int *>(sm + L * F::P);
  double *base = d.field[blockIdx.y];
  const long long row0 = (long long)blockIdx.x * 16;
  if (t < 8) emax[t] = 0;
  __syncthreads();
  for (int q = t >> 5; q < 16; q += W) {
    const long long row = row0 + q;
    const bool lv = row < d.rows;
    const double *src = base + row * d.pitch;
    const int p = q >> 1, second = q & 1;
    int em = 0;
    constexpr int NL = (L + 31) / 32;
    double v[NL];
#pragma unroll
    for (int c = 0; c < NL; ++c) {
      const int e = lane + 32 * c;
      v[c] = 0.0;
      if (lv && (L % 32 == 0 || e < L)) v[c] = src[e];
    }
#pragma unroll
    for (int c = 0; c < NL; ++c) {
      const int e = lane + 32 * c;
      if (L % 32 == 0 || e < L) {
        em = max(em, dbl_exponent(v[c]));
        reinterpret_cast<double *>(&sm[F::slot(e, p)])[second] = v[c];
      }
    }
    em = int(__reduce_max_sync(0xffffffffu, unsigned(em)));
    if (lane == 0) atomicMax(&emax[p], em);
  }
  __syncthreads();
  {
    const int sh = emax[pen] + 63 - a.B;
    typename F::template Regs<0> g;
    F::template load<0>(g, sm, pen);
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
#pragma unroll
        for (int r = 0; r < F::D::R(0); ++r)
          g.v[m][r] = {to_fixed(__longlong_as_double(g.v[m][r].x), sh), to_fixed(__longlong_as_double(g.v[m][r].y), sh)};
      }
    F::template butterfly<0>(g, a.tw);
    __syncthreads();
    F::template store<0>(g, sm, pen);
    __syncthreads();
  }
  F::template rest<1>(sm, pen, a.tw, [&](auto &g) {
    __syncthreads();
    F::template store<F::last>(g, sm, pen);
    __syncthreads();
  });
  const int kc = d.kc;
  for (int q = t >> 5; q < 16; q += W) {
    const long long row = row0 + q;
    if (row >= d.rows) break;
    double2 *dst = reinterpret_cast<double2 *>(base + row * d.pitch);
    const int p = q >> 1, second = q & 1;
    const int S = emax[p] - 1022 - a.B + 3 * (F::steps - 1) - 1;
    const bool bad = emax[p] == 2047;
#pragma unroll 2
    for (int k = lane; k < kc; k += 32) {
      const longlong2 u = sm[F::slot(k, p)], w = sm[F::slot(k ? L - k : 0, p)];
      const long long x = second ? u.y + w.y : u.x + w.x, y = second ? w.x - u.x : u.y - w.y;
      dst[k] = bad ? make_double2(nan_of(), nan_of()) : make_double2(to_double(x, S), to_double(y, S));
    }
  }
}

// what of a length is launched
enum FxOp { FX_OP_PREPARE = 0, FX_OP_STRIDED, FX_OP_TRUNCATE, FX_OP_C2R, FX_OP_R2C };

template <int L> cudaError_t launch_len(FxOp op, const void *args, dim3 grid, cudaStream_t st) {
  using F = Fft<L>;
  switch (op) {
    case FX_OP_PREPARE: {
      cudaError_t e = cudaSuccess;
      for (const void *f : {(const void *)k_fx_strided_l<L, false>, (const void *)k_fx_strided_l<L, true>,
                            (const void *)k_fx_c2r_l<L>, (const void *)k_fx_r2c_l<L>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, F::smem);
      return e;
    }
    case FX_OP_STRIDED: k_fx_strided_l<L, false><<<grid, F::T, F::smem, st>>>(*static_cast<const LArgs *>(args)); break;
    case FX_OP_TRUNCATE: k_fx_strided_l<L, true><<<grid, F::T, F::smem, st>>>(*static_cast<const LArgs *>(args)); break;
    case FX_OP_C2R: k_fx_c2r_l<L><<<grid, F::T, F::smem, st>>>(*static_cast<const LRows *>(args)); break;
    case FX_OP_R2C: k_fx_r2c_l<L><<<grid, F::T, F::smem, st>>>(*static_cast<const LRows *>(args)); break;
  }
  return cudaGetLastError();
}

}  // namespace fx
