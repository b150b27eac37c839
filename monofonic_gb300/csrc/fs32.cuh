// Pruned pencil transforms of single-precision fields: the FP32 form's grids
// that the fused transforms (fused.cuh) are not built for -- padded lengths
// without an instance there, noise that fills the Nyquist planes, 1LPT.
//
// The passes are those of the plain FP64 form (fx64.h, fx64_len.cuh): rows that
// the Orszag padding makes zero are neither read, transformed nor written, the
// Hessian factors, the inverse Laplacian and convolve3's truncation are applied
// while loading and storing.  HBM bounds them (a pencil point is 8 bytes read and
// 8 written against about 100 instructions); a CTA holds 16 pencils of adjacent
// kz, 128-byte row pieces, in shared memory and exchanges through it once for two
// steps.  cuFFT ran the same transforms at 1.0 TB/s of field traffic (3 passes
// each, unpruned): 256^3 MUSIC1 3LPT 12.4 ms of an 18.1 ms pass.
#pragma once
#include "fx64.cuh"
#include "fx64.h"

namespace fx {

// radices of a length in the order of a forward transform (the last divisible
// by three where the length serves as padded length), threads of 16 pencils
template <int L> struct Len32;
#define FS_LEN(L_, STEPS_, A_, B_, C_, T_, CTAS_)                             \
  template <> struct Len32<L_> {                                             \
    static constexpr int steps = STEPS_, T = T_, ctas = CTAS_;                \
    static FX_HD constexpr int R(int q) { return q == 0 ? A_ : (q == 1 ? B_ : C_); } \
  };
FS_LEN(16, 2, 4, 4, 1, 64, 8)
FS_LEN(24, 2, 4, 6, 1, 96, 8)
FS_LEN(32, 2, 4, 8, 1, 128, 6)
FS_LEN(48, 2, 8, 6, 1, 128, 6)
FS_LEN(64, 2, 8, 8, 1, 128, 6)
FS_LEN(96, 2, 8, 12, 1, 192, 4)
FS_LEN(128, 2, 8, 16, 1, 256, 3)
FS_LEN(192, 2, 16, 12, 1, 256, 3)
FS_LEN(256, 2, 16, 16, 1, 256, 3)
FS_LEN(384, 2, 16, 24, 1, 384, 2)
FS_LEN(512, 3, 8, 8, 8, 512, 2)
FS_LEN(768, 3, 8, 8, 12, 512, 2)
FS_LEN(56, 2, 7, 8, 1, 128, 6)
FS_LEN(60, 2, 10, 6, 1, 160, 5)
FS_LEN(80, 2, 8, 10, 1, 160, 5)
FS_LEN(84, 2, 7, 12, 1, 192, 4)
FS_LEN(90, 2, 10, 9, 1, 160, 5)
FS_LEN(100, 2, 10, 10, 1, 160, 5)
FS_LEN(108, 2, 9, 12, 1, 192, 4)
FS_LEN(112, 2, 8, 14, 1, 224, 3)
FS_LEN(120, 2, 10, 12, 1, 192, 4)
FS_LEN(126, 2, 14, 9, 1, 224, 3)
FS_LEN(140, 2, 10, 14, 1, 224, 3)
FS_LEN(150, 2, 10, 15, 1, 256, 3)
FS_LEN(160, 2, 10, 16, 1, 256, 3)
FS_LEN(162, 2, 9, 18, 1, 288, 2)
FS_LEN(168, 2, 14, 12, 1, 224, 3)
FS_LEN(180, 2, 15, 12, 1, 256, 3)
FS_LEN(196, 2, 14, 14, 1, 224, 3)
FS_LEN(200, 2, 10, 20, 1, 320, 2)
FS_LEN(210, 2, 14, 15, 1, 256, 3)
FS_LEN(216, 2, 12, 18, 1, 288, 2)
FS_LEN(224, 2, 14, 16, 1, 256, 3)
FS_LEN(240, 2, 16, 15, 1, 256, 3)
FS_LEN(252, 2, 14, 18, 1, 288, 2)
FS_LEN(270, 2, 15, 18, 1, 288, 2)
FS_LEN(294, 2, 14, 21, 1, 352, 2)
FS_LEN(300, 2, 20, 15, 1, 320, 2)
FS_LEN(324, 2, 18, 18, 1, 288, 2)
FS_LEN(336, 2, 14, 24, 1, 384, 2)
FS_LEN(360, 2, 20, 18, 1, 320, 2)
FS_LEN(378, 2, 18, 21, 1, 352, 2)
FS_LEN(72, 2, 8, 9, 1, 160, 5)
FS_LEN(144, 2, 12, 12, 1, 192, 4)
#undef FS_LEN

__device__ __forceinline__ F2 ld(const float2 *p) {
  const float2 v = *p;
  return {v.x, v.y};
}
__device__ __forceinline__ F2 cmul(F2 v, float2 w) { return {v.x * w.x - v.y * w.y, v.x * w.y + v.y * w.x}; }
__device__ __forceinline__ F2 swap_if(F2 v, bool s) { return s ? F2{v.y, v.x} : v; }

template <int L, bool REV> struct Fft32 {
  using D = Len32<L>;
  static constexpr int P = 16, lgP = 4, T = D::T, steps = D::steps, W = T / 32, last = D::steps - 1;
  static constexpr int smem = L * P * 8;
  static FX_HD constexpr int R(int q) { return D::R(REV ? steps - 1 - q : q); }
  static FX_HD constexpr int NS(int q) { return q == 0 ? 1 : NS(q - 1) * R(q - 1); }
  static FX_HD constexpr int MU(int q) { return (P * (L / R(q)) + T - 1) / T; }
  static __device__ __forceinline__ int slot(int e, int pen) { return (e << lgP) + (pen ^ (e & (P - 1))); }
  template <int Q> struct Regs {
    F2 v[MU(Q)][R(Q)];
  };
  template <int Q> static __device__ __forceinline__ bool live(int m) {
    constexpr int items = P * (L / R(Q));
    return items % T == 0 || int(threadIdx.x) + m * T < items;
  }
  template <int Q> static __device__ __forceinline__ int jof(int m) { return (int(threadIdx.x) + m * T) >> lgP; }
  template <int Q> static __device__ __forceinline__ int out_of(int j, int r) {
    constexpr int ns = NS(Q);
    return (j / ns) * (ns * R(Q)) + j % ns + r * ns;
  }
  template <int Q> static __device__ __forceinline__ void load(Regs<Q> &g, const F2 *s, int pen) {
#pragma unroll
    for (int m = 0; m < MU(Q); ++m)
      if (live<Q>(m)) {
        const int j = jof<Q>(m);
#pragma unroll
        for (int r = 0; r < R(Q); ++r) g.v[m][r] = s[slot(j + r * (L / R(Q)), pen)];
      }
  }
  // outputs r of FROM < r < TO are left out
  template <int Q, int FROM = 0, int TO = 0>
  static __device__ __forceinline__ void store(const Regs<Q> &g, F2 *s, int pen) {
#pragma unroll
    for (int m = 0; m < MU(Q); ++m)
      if (live<Q>(m)) {
        const int j = jof<Q>(m);
#pragma unroll
        for (int r = 0; r < R(Q); ++r)
          if (!(r > FROM && r < TO)) s[slot(out_of<Q>(j, r), pen)] = g.v[m][r];
      }
  }
  template <int Q> static __device__ __forceinline__ void butterfly(Regs<Q> &g, const float2 *tw) {
    constexpr int ns = NS(Q);
#pragma unroll
    for (int m = 0; m < MU(Q); ++m)
      if (live<Q>(m)) {
        if constexpr (Q > 0) {
          const int inc = (jof<Q>(m) % ns) * (L / (ns * R(Q)));
#pragma unroll
          for (int r = 1; r < R(Q); ++r) g.v[m][r] = cmul(g.v[m][r], __ldg(&tw[r * inc]));
        }
        Dft<R(Q)>::run(g.v[m]);
      }
  }
  template <int Q, class F> static __device__ __forceinline__ void rest(F2 *s, int pen, const float2 *tw, F &&out) {
    Regs<Q> g;
    load<Q>(g, s, pen);
    butterfly<Q>(g, tw);
    if constexpr (Q + 1 < steps) {
      __syncthreads();
      store<Q>(g, s, pen);
      __syncthreads();
      rest<Q + 1>(s, pen, tw, out);
    } else {
      out(g);
    }
  }
};

// zones of the padded positions, as in fx64_len.cuh
enum Zone32 { S_LOW, S_NYQ, S_PAD, S_EDGE, S_HIGH };
template <int R> FX_HD constexpr Zone32 zone32(int r) {
  return r < R / 3 ? S_LOW : (r == R / 3 ? S_NYQ : (r < 2 * R / 3 ? S_PAD : (r == 2 * R / 3 ? S_EDGE : S_HIGH)));
}

// factor (row index)^pr (kz)^pk in_fac of an input, Nyquist zero
__device__ __forceinline__ float row_factor(int i, int n, int pr) {
  const float f = i == (n >> 1) ? 0.f : float(i > (n >> 1) ? i - n : i);
  return pr == 0 ? 1.f : (pr == 1 ? f : f * f);
}
__device__ __forceinline__ float kz_factor(int kz, int n, int pk, double in_fac) {
  const float k = kz == (n >> 1) ? 0.f : float(kz), f = in_fac != 0.0 ? float(in_fac) : 1.f;
  return pk == 0 ? f : (pk == 1 ? k * f : k * k * f);
}

// inverse transform along x or y; PAD: N rows in, placed at the padded positions
template <int L, bool PAD>
__global__ void __launch_bounds__(Len32<L>::T, Len32<L>::ctas) k_fs_inv(const __grid_constant__ Strided d) {
  mfx::pdl_begin();
  using F = Fft32<L, true>;
  extern __shared__ __align__(16) F2 fsm[];
  constexpr int R0 = F::R(0), nb = L / R0, nh = L / 3, n = 2 * nh;
  const int t = threadIdx.x, pen = t & 15;
  const float2 *tw = static_cast<const float2 *>(d.tw);
  const int kblocks = (d.kc + 15) >> 4;
  const int o = blockIdx.x / kblocks, kz = ((blockIdx.x - o * kblocks) << 4) + pen;
  const bool lv = kz < d.kc;
  for (int op = d.first[blockIdx.y]; op < d.first[blockIdx.y + 1]; ++op) {
    const float2 *src = static_cast<const float2 *>(d.src[op]) + (long long)o * d.in_outer + kz;
    const int pr = d.pr[op];
    const bool scaled = PAD && ((pr | d.pk[op]) != 0 || d.in_fac != 0.0);
    const float kf = PAD ? kz_factor(kz, n, d.pk[op], d.in_fac) : 1.f;
    typename F::template Regs<0> g;
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
        const int j = F::template jof<0>(m);
        const float2 *p = src + (long long)j * d.in_row;
        const long long stride = (long long)nb * d.in_row, back = PAD ? (long long)nh * d.in_row : 0;
#pragma unroll
        for (int r = 0; r < R0; ++r) {
          const Zone32 z = PAD ? zone32<R0>(r) : S_LOW;
          g.v[m][r] = {0.f, 0.f};
          if (z == S_PAD) continue;
          if (lv && (z == S_NYQ ? j == 0 : (z == S_EDGE ? j > 0 : true)))
            g.v[m][r] = swap_if(ld(p + r * stride - (z >= S_EDGE ? back : 0)), true);
        }
        if (scaled) {
#pragma unroll
          for (int r = 0; r < R0; ++r) {
            const Zone32 z = zone32<R0>(r);
            if (z == S_PAD) continue;
            const float f = row_factor(j + r * nb - (z >= S_EDGE ? nh : 0), n, pr) * kf;
            g.v[m][r] = {g.v[m][r].x * f, g.v[m][r].y * f};
          }
        }
      }
    F::template butterfly<0>(g, tw);
    F::template store<0>(g, fsm, pen);
    __syncthreads();
    float2 *dst = static_cast<float2 *>(d.dst[op]) + (long long)o * d.out_outer + kz;
    F::template rest<1>(fsm, pen, tw, [&](auto &h) {
      constexpr int Q = F::last;
#pragma unroll
      for (int m = 0; m < F::MU(Q); ++m)
        if (F::template live<Q>(m) && lv) {
          float2 *p = dst + (long long)F::template jof<Q>(m) * d.out_row;
          const long long stride = (long long)F::NS(Q) * d.out_row;
#pragma unroll
          for (int r = 0; r < F::R(Q); ++r) p[r * stride] = make_float2(h.v[m][r].y, h.v[m][r].x);
        }
    });
    if (op + 1 < d.first[blockIdx.y + 1]) __syncthreads();
  }
}

// the N-grid rows of a transformed pencil, times -fac / k^2 with inv_lap
__device__ __forceinline__ float lap_factor(const Strided &d, int so, int si, int kz) {
  const int q = so * so + si * si + kz * kz;
  return q ? -float(d.fac) / float(q) : 0.f;
}

// forward transform along x or y, the N-grid rows kept (the Nyquist row zero)
template <int L> __global__ void __launch_bounds__(Len32<L>::T, Len32<L>::ctas) k_fs_cut(const __grid_constant__ Strided d) {
  mfx::pdl_begin();
  using F = Fft32<L, false>;
  extern __shared__ __align__(16) F2 fsm[];
  constexpr int R0 = F::R(0), nb = L / R0, nh = L / 3, n = 2 * nh;
  const int t = threadIdx.x, pen = t & 15;
  const float2 *tw = static_cast<const float2 *>(d.tw);
  const int kblocks = (d.kc + 15) >> 4;
  const int o = blockIdx.x / kblocks, kz0 = (blockIdx.x - o * kblocks) << 4, kz = kz0 + pen, op = blockIdx.y;
  const bool lv = kz < d.kc;
  const float2 *src = static_cast<const float2 *>(d.src[op]) + (long long)o * d.in_outer + kz;
  typename F::template Regs<0> g;
#pragma unroll
  for (int m = 0; m < F::MU(0); ++m)
    if (F::template live<0>(m)) {
      const float2 *p = src + (long long)F::template jof<0>(m) * d.in_row;
      const long long stride = (long long)nb * d.in_row;
#pragma unroll
      for (int r = 0; r < R0; ++r) {
        g.v[m][r] = {0.f, 0.f};
        if (lv) g.v[m][r] = ld(p + r * stride);
      }
    }
  F::template butterfly<0>(g, tw);
  F::template store<0>(g, fsm, pen);
  __syncthreads();
  float2 *dst = static_cast<float2 *>(d.dst[op]) + (long long)o * d.out_outer + kz;
  F::template rest<1>(fsm, pen, tw, [&](auto &h) {
    constexpr int Q = F::last, RL = F::R(Q);
    const int so = o > nh ? o - n : o;
#pragma unroll
    for (int m = 0; m < F::MU(Q); ++m)
      if (F::template live<Q>(m) && lv) {
        const int j = F::template jof<Q>(m);
        float2 *p = dst + (long long)j * d.out_row;
        const long long stride = (long long)F::NS(Q) * d.out_row, back = (long long)nh * d.out_row;
#pragma unroll
        for (int r = 0; r < RL; ++r) {
          const Zone32 z = zone32<RL>(r);
          if (z == S_PAD || (z == S_NYQ && j != 0) || (z == S_EDGE && j == 0)) continue;
          float2 v = make_float2(0.f, 0.f);
          if (z != S_NYQ) {
            v = make_float2(h.v[m][r].x, h.v[m][r].y);
            if (d.inv_lap) {
              const float f = o == nh ? 0.f : lap_factor(d, so, j + r * (L / RL) - (z >= S_EDGE ? L : 0), kz);
              v.x *= f;
              v.y *= f;
            }
          }
          *(p + r * stride - (z >= S_EDGE ? back : 0)) = v;
        }
      }
  });
  if (d.inv_lap && kz0 + 16 >= d.kc) {
    float2 *z = static_cast<float2 *>(d.dst[op]) + (long long)o * d.out_outer + d.kc;  // the kz Nyquist column
    for (int i = t; i < n; i += F::T) z[(long long)i * d.out_row] = make_float2(0.f, 0.f);
  }
}

// forward, the N-grid rows kept times fac, and back (in place)
template <int L>
__global__ void __launch_bounds__(Len32<L>::T, Len32<L>::ctas) k_fs_trunc(const __grid_constant__ Strided d) {
  mfx::pdl_begin();
  using F = Fft32<L, false>;
  using I = Fft32<L, true>;
  extern __shared__ __align__(16) F2 fsm[];
  constexpr int R0 = F::R(0), nb = L / R0, RL = F::R(F::last);
  static_assert(RL == I::R(0), "the forward transform's last radix is the inverse one's first");
  const int t = threadIdx.x, pen = t & 15;
  const float2 *tw = static_cast<const float2 *>(d.tw);
  const int kblocks = (d.kc + 15) >> 4;
  const int o = blockIdx.x / kblocks, kz = ((blockIdx.x - o * kblocks) << 4) + pen, op = blockIdx.y;
  const bool lv = kz < d.kc;
  const float fac = float(d.fac);
  typename I::template Regs<0> h;
  {
    const float2 *src = static_cast<const float2 *>(d.src[op]) + (long long)o * d.in_outer + kz;
    typename F::template Regs<0> g;
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
        const float2 *p = src + (long long)F::template jof<0>(m) * d.in_row;
        const long long stride = (long long)nb * d.in_row;
#pragma unroll
        for (int r = 0; r < R0; ++r) {
          g.v[m][r] = {0.f, 0.f};
          if (lv) g.v[m][r] = ld(p + r * stride);
        }
      }
    F::template butterfly<0>(g, tw);
    F::template store<0>(g, fsm, pen);
    __syncthreads();
  }
  F::template rest<1>(fsm, pen, tw, [&](auto &g) {
#pragma unroll
    for (int m = 0; m < F::MU(F::last); ++m)
      if (F::template live<F::last>(m)) {
        const int j = F::template jof<F::last>(m);
#pragma unroll
        for (int r = 0; r < RL; ++r) {
          const Zone32 z = zone32<RL>(r);
          const F2 v = g.v[m][r];
          h.v[m][r] = (z == S_NYQ || z == S_PAD || (z == S_EDGE && j == 0)) ? F2{0.f, 0.f} : F2{v.y * fac, v.x * fac};
        }
      }
  });
  __syncthreads();
  I::template butterfly<0>(h, tw);
  I::template store<0>(h, fsm, pen);
  __syncthreads();
  float2 *dst = static_cast<float2 *>(d.dst[op]) + (long long)o * d.out_outer + kz;
  I::template rest<1>(fsm, pen, tw, [&](auto &g) {
    constexpr int Q = I::last;
#pragma unroll
    for (int m = 0; m < I::MU(Q); ++m)
      if (I::template live<Q>(m) && lv) {
        float2 *p = dst + (long long)I::template jof<Q>(m) * d.out_row;
        const long long stride = (long long)I::NS(Q) * d.out_row;
#pragma unroll
        for (int r = 0; r < I::R(Q); ++r) p[r * stride] = make_float2(g.v[m][r].y, g.v[m][r].x);
      }
  });
}

// spectra -> real rows, two rows a pencil: Z[k] = A[k] + i B[k], Z[L - k] =
// conj A[k] + i conj B[k]; PAD: at most L/3 + 1 kz values
template <int L, bool PAD>
__global__ void __launch_bounds__(Len32<L>::T, Len32<L>::ctas) k_fs_c2r(const __grid_constant__ Rows d) {
  mfx::pdl_begin();
  using F = Fft32<L, true>;
  extern __shared__ __align__(16) F2 fsm[];
  constexpr int h = L / 2, kmax = PAD ? L / 3 + 1 : h, NL = (kmax + 31) / 32;
  const int t = threadIdx.x, lane = t & 31, pen = t & 15;
  const float2 *tw = static_cast<const float2 *>(d.tw);
  float *base = static_cast<float *>(d.field[blockIdx.y]);
  const long long row0 = (long long)blockIdx.x * 32;
  const int kc = min(d.kc, kmax);
  // a warp takes both rows of a pencil and writes its exchanged spectrum
#pragma unroll 1
  for (int p = t >> 5; p < 16; p += F::W) {
    const long long row = row0 + 2 * p;
    const bool la = row < d.rows, lb = row + 1 < d.rows;
    const float2 *sa = reinterpret_cast<const float2 *>(base + row * d.pitch);
    const float2 *sb = reinterpret_cast<const float2 *>(base + (row + 1) * d.pitch);
    F2 a[NL], b[NL];
#pragma unroll
    for (int c = 0; c < NL; ++c) {
      const int k = lane + 32 * c;
      a[c] = b[c] = {0.f, 0.f};
      if (la && k < kc) a[c] = ld(sa + k);
      if (lb && k < kc) b[c] = ld(sb + k);
    }
#pragma unroll
    for (int c = 0; c < NL; ++c) {
      const int k = lane + 32 * c;
      if (k >= kmax) continue;
      if (k == 0) {
        fsm[F::slot(0, p)] = {b[c].x, a[c].x};  // only the real part of the k = 0 value is used
        continue;
      }
      fsm[F::slot(k, p)] = {a[c].y + b[c].x, a[c].x - b[c].y};
      fsm[F::slot(L - k, p)] = {b[c].x - a[c].y, a[c].x + b[c].y};
    }
    if (!PAD && lane == 0) {
      const bool nyq = d.kc > h;  // zero where the spectrum ends before it
      fsm[F::slot(h, p)] = {nyq && lb ? sb[h].x : 0.f, nyq && la ? sa[h].x : 0.f};
    }
  }
  __syncthreads();
  {
    typename F::template Regs<0> g;
    constexpr int R0 = F::R(0), nb = L / R0;
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
        const int j = F::template jof<0>(m);
#pragma unroll
        for (int r = 0; r < R0; ++r) {
          const Zone32 z = PAD ? zone32<R0>(r) : S_LOW;
          g.v[m][r] = {0.f, 0.f};
          if (z == S_PAD || (z == S_NYQ && j != 0)) continue;
          g.v[m][r] = fsm[F::slot(j + r * nb, pen)];
        }
      }
    F::template butterfly<0>(g, tw);
    __syncthreads();
    F::template store<0>(g, fsm, pen);
    __syncthreads();
  }
  F::template rest<1>(fsm, pen, tw, [&](auto &g) {
    __syncthreads();
    F::template store<F::last>(g, fsm, pen);
    __syncthreads();
  });
#pragma unroll 1
  for (int p = t >> 5; p < 16; p += F::W) {
    const long long row = row0 + 2 * p;
    float *da = base + row * d.pitch, *db = da + d.pitch;
    const bool la = row < d.rows, lb = row + 1 < d.rows;
#pragma unroll 4
    for (int e = lane; e < L; e += 32) {
      const F2 v = fsm[F::slot(e, p)];  // exchanged again: the first row is the imaginary part
      if (la) da[e] = v.y;
      if (lb) db[e] = v.x;
    }
  }
}

// real rows -> spectra of kz < kc <= L/3
template <int L> __global__ void __launch_bounds__(Len32<L>::T, Len32<L>::ctas) k_fs_r2c(const __grid_constant__ Rows d) {
  mfx::pdl_begin();
  using F = Fft32<L, false>;
  extern __shared__ __align__(16) F2 fsm[];
  constexpr int NL = (L + 31) / 32;
  const int t = threadIdx.x, lane = t & 31, pen = t & 15;
  const float2 *tw = static_cast<const float2 *>(d.tw);
  float *base = static_cast<float *>(d.field[blockIdx.y]);
  const long long row0 = (long long)blockIdx.x * 32;
#pragma unroll 1
  for (int p = t >> 5; p < 16; p += F::W) {
    const long long row = row0 + 2 * p;
    const bool la = row < d.rows, lb = row + 1 < d.rows;
    const float *sa = base + row * d.pitch, *sb = sa + d.pitch;
    F2 v[NL];
#pragma unroll
    for (int c = 0; c < NL; ++c) {
      const int e = lane + 32 * c;
      v[c] = {0.f, 0.f};
      if (L % 32 == 0 || e < L) {
        if (la) v[c].x = sa[e];
        if (lb) v[c].y = sb[e];
      }
    }
#pragma unroll
    for (int c = 0; c < NL; ++c) {
      const int e = lane + 32 * c;
      if (L % 32 == 0 || e < L) fsm[F::slot(e, p)] = v[c];
    }
  }
  __syncthreads();
  {
    typename F::template Regs<0> g;
    F::template load<0>(g, fsm, pen);
    F::template butterfly<0>(g, tw);
    __syncthreads();
    F::template store<0>(g, fsm, pen);
    __syncthreads();
  }
  F::template rest<1>(fsm, pen, tw, [&](auto &g) {
    constexpr int RL = F::R(F::last);
    __syncthreads();
    F::template store<F::last, RL / 3 - 1, 2 * RL / 3>(g, fsm, pen);
    __syncthreads();
  });
  const int kc = d.kc;
#pragma unroll 1
  for (int p = t >> 5; p < 16; p += F::W) {
    const long long row = row0 + 2 * p;
    float2 *da = reinterpret_cast<float2 *>(base + row * d.pitch), *db = reinterpret_cast<float2 *>(base + (row + 1) * d.pitch);
    const bool la = row < d.rows, lb = row + 1 < d.rows;
#pragma unroll 2
    for (int k = lane; k < kc; k += 32) {
      const F2 u = fsm[F::slot(k, p)], w = fsm[F::slot(k ? L - k : 0, p)];
      // A = (Z[k] + conj Z[L-k]) / 2, B = (Z[k] - conj Z[L-k]) / 2i
      if (la) da[k] = make_float2(0.5f * (u.x + w.x), 0.5f * (u.y - w.y));
      if (lb) db[k] = make_float2(0.5f * (u.y + w.y), 0.5f * (w.x - u.x));
    }
  }
}

enum FsOp { FS_PREPARE = 0, FS_INV_PAD, FS_CUT, FS_TRUNC, FS_C2R_PAD, FS_R2C, FS_INV, FS_C2R };

// (defined outside the class: an inline member would be instantiated, kernels and
// all, wherever its address is taken)
template <int L, bool PADDED, bool GRID> struct Launch32 {
  static cudaError_t run(FsOp op, const Strided *s, const Rows *r, dim3 grid, cudaStream_t st);
};
template <int L, bool PADDED, bool GRID>
cudaError_t Launch32<L, PADDED, GRID>::run(FsOp op, const Strided *s, const Rows *r, dim3 grid, cudaStream_t st) {
  using F = Fft32<L, false>;
  cudaError_t e = cudaSuccess;
  auto limit = [&](const void *f) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, F::smem);
  };
  bool done = op == FS_PREPARE;
  if constexpr (PADDED) {
    if (op == FS_PREPARE) {
      limit((const void *)k_fs_inv<L, true>);
      limit((const void *)k_fs_cut<L>);
      limit((const void *)k_fs_trunc<L>);
      limit((const void *)k_fs_c2r<L, true>);
      limit((const void *)k_fs_r2c<L>);
    }
    done = true;
    if (op == FS_INV_PAD) mfx::launch_pdl(k_fs_inv<L, true>, grid, F::T, F::smem, st, *s);
    else if (op == FS_CUT) mfx::launch_pdl(k_fs_cut<L>, grid, F::T, F::smem, st, *s);
    else if (op == FS_TRUNC) mfx::launch_pdl(k_fs_trunc<L>, grid, F::T, F::smem, st, *s);
    else if (op == FS_C2R_PAD) mfx::launch_pdl(k_fs_c2r<L, true>, grid, F::T, F::smem, st, *r);
    else if (op == FS_R2C) mfx::launch_pdl(k_fs_r2c<L>, grid, F::T, F::smem, st, *r);
    else done = op == FS_PREPARE;
  }
  if constexpr (GRID) {
    if (op == FS_PREPARE) {
      limit((const void *)k_fs_inv<L, false>);
      limit((const void *)k_fs_c2r<L, false>);
    }
    if (op == FS_INV) {
      mfx::launch_pdl(k_fs_inv<L, false>, grid, F::T, F::smem, st, *s);
      done = true;
    } else if (op == FS_C2R) {
      mfx::launch_pdl(k_fs_c2r<L, false>, grid, F::T, F::smem, st, *r);
      done = true;
    }
  }
  if (!done) return cudaErrorInvalidValue;
  return e == cudaSuccess ? cudaGetLastError() : e;
}

}  // namespace fx
