// The fixed-point transforms (fx64.cuh) compiled for one length: radices, index
// arithmetic and thread counts are constants, the first step of an x or y pass
// reads HBM straight into registers and the last one writes from them (one
// shared-memory exchange for two steps).  Lengths without an instance take the
// run-time kernels of fx64.cu.
//
// What bounds them: at 384 the ALU pipe is 54% busy in the z passes (FP64, the
// conversions back, 20 - 30%, HBM 30%), 37% in the x and y passes (FP64 45%, HBM 20 -
// 25%), the rest is latency at the 12 - 18 warps that their registers leave an SM.
// So what they save is instructions.
//  * A padded length L = 3N/2 is split so that the step at its N-grid side (the
//    first of an inverse transform, the last of a forward one) has a radix
//    divisible by three: inputs r of R / 3 < r < 2R / 3 of that step are the
//    padding, for every butterfly, and neither loaded, converted, added nor
//    stored.
//  * In convolve3's truncation the forward transform's last step and the
//    inverse one's first step have the same radix: the butterflies' outputs
//    are the next ones' inputs and stay in registers.
//  * Twiddles are read as the three constants of the complex product, split
//    for the 32-bit multiplications.
#pragma once
#include "fx64.cuh"
#include "fx64.h"

namespace fx {

// radices of a length in the order of a forward transform (an inverse one takes
// them backwards), threads per CTA of eight pencils, CTAs an SM is to hold
template <int L> struct Len;
#define FX_LEN(L_, STEPS_, A_, B_, C_, T_, CTAS_, ZCTAS_)                     \
  template <> struct Len<L_> {                                               \
    static constexpr int steps = STEPS_, T = T_, ctas = CTAS_, zctas = ZCTAS_; \
    static FX_HD constexpr int R(int q) { return q == 0 ? A_ : (q == 1 ? B_ : C_); } \
  };
FX_LEN(16, 2, 4, 4, 1, 32, 12, 16)
FX_LEN(24, 2, 4, 6, 1, 64, 8, 12)
FX_LEN(32, 2, 4, 8, 1, 64, 8, 12)
FX_LEN(48, 2, 8, 6, 1, 64, 8, 12)
FX_LEN(64, 2, 8, 8, 1, 64, 8, 12)
FX_LEN(72, 2, 8, 9, 1, 96, 5, 8)
FX_LEN(96, 2, 8, 12, 1, 96, 5, 8)
FX_LEN(128, 2, 8, 16, 1, 128, 4, 5)
FX_LEN(144, 2, 12, 12, 1, 96, 5, 7)
FX_LEN(192, 2, 16, 12, 1, 128, 4, 5)
FX_LEN(256, 2, 16, 16, 1, 128, 4, 5)
FX_LEN(288, 2, 16, 18, 1, 160, 3, 4)
FX_LEN(384, 2, 16, 24, 1, 192, 2, 3)
FX_LEN(512, 3, 8, 8, 8, 256, 2, 2)
FX_LEN(576, 2, 24, 24, 1, 192, 2, 3)
FX_LEN(768, 3, 8, 8, 12, 256, 2, 2)
FX_LEN(1152, 3, 8, 12, 12, 384, 1, 1)
// the other grids from 56 to 252 with prime factors up to 7 and their padded
// lengths (100^3 BCC 3LPT: 3.54 ms with the run-time kernels, 2.28 ms with these)
FX_LEN(56, 2, 7, 8, 1, 64, 7, 10)
FX_LEN(60, 2, 10, 6, 1, 96, 5, 6)
FX_LEN(80, 2, 8, 10, 1, 96, 5, 6)
FX_LEN(84, 2, 7, 12, 1, 96, 5, 6)
FX_LEN(90, 2, 10, 9, 1, 96, 5, 6)
FX_LEN(100, 2, 10, 10, 1, 96, 5, 6)
FX_LEN(108, 2, 9, 12, 1, 96, 5, 6)
FX_LEN(112, 2, 8, 14, 1, 128, 3, 5)
FX_LEN(120, 2, 10, 12, 1, 96, 5, 6)
FX_LEN(126, 2, 14, 9, 1, 128, 3, 5)
FX_LEN(140, 2, 10, 14, 1, 128, 3, 5)
FX_LEN(150, 2, 10, 15, 1, 128, 3, 5)
FX_LEN(160, 2, 10, 16, 1, 128, 3, 5)
FX_LEN(162, 2, 9, 18, 1, 160, 3, 4)
FX_LEN(168, 2, 14, 12, 1, 128, 3, 5)
FX_LEN(180, 2, 15, 12, 1, 128, 3, 5)
FX_LEN(196, 2, 14, 14, 1, 128, 3, 5)
FX_LEN(200, 2, 10, 20, 1, 160, 3, 4)
FX_LEN(210, 2, 14, 15, 1, 128, 3, 5)
FX_LEN(216, 2, 12, 18, 1, 160, 3, 4)
FX_LEN(224, 2, 14, 16, 1, 128, 3, 5)
FX_LEN(240, 2, 16, 15, 1, 128, 3, 5)
FX_LEN(252, 2, 14, 18, 1, 160, 3, 4)
FX_LEN(270, 2, 15, 18, 1, 160, 3, 4)
FX_LEN(294, 2, 14, 21, 1, 192, 2, 3)
FX_LEN(300, 2, 20, 15, 1, 160, 3, 4)
FX_LEN(324, 2, 18, 18, 1, 160, 3, 4)
FX_LEN(336, 2, 14, 24, 1, 192, 2, 3)
FX_LEN(360, 2, 20, 18, 1, 160, 3, 4)
FX_LEN(378, 2, 18, 21, 1, 192, 2, 3)
#undef FX_LEN
// the instances: length, as padded length, as grid length
#define FX_LENGTHS(X) \
  X(16, false, true) X(24, true, true) X(32, false, true) X(48, true, true) X(64, false, true) X(72, true, true) \
  X(96, true, true) X(128, false, true) X(144, true, true) X(192, true, true) X(256, false, true) \
  X(288, true, false) X(384, true, true) X(512, false, true) X(576, true, false) X(768, true, true) \
  X(1152, true, false) X(56, false, true) X(60, false, true) X(80, false, true) X(84, true, true) \
  X(90, true, false) X(100, false, true) X(108, true, true) X(112, false, true) X(120, true, true) \
  X(126, true, false) X(140, false, true) X(150, true, false) X(160, false, true) X(162, true, false) \
  X(168, true, true) X(180, true, true) X(196, false, true) X(200, false, true) X(210, true, false) \
  X(216, true, true) X(224, false, true) X(240, true, true) X(252, true, true) X(270, true, false) \
  X(294, true, false) X(300, true, false) X(324, true, false) X(336, true, false) X(360, true, false) \
  X(378, true, false)

// the constants of the twiddle products (fx64.cuh twiddle4) of a length
struct Tw3 {
  const int4 *cp;  // c: hi, lo; s + c: hi, lo
  const int2 *m;   // s - c: hi, lo
};
__device__ __forceinline__ Tw3 tw3_of(const void *table, int L) {
  const int4 *cp = static_cast<const int4 *>(table);
  return {cp, reinterpret_cast<const int2 *>(cp + L)};
}
__device__ __forceinline__ I2 twiddle4(I2 v, const Tw3 &t, int at) { return twiddle4(v, __ldg(&t.cp[at]), __ldg(&t.m[at])); }

// high word without the sign: its maximum has the largest exponent
__device__ __forceinline__ int mag(long long b) { return int(b >> 32) & 0x7fffffff; }
// the larger component's of a value that is still a double; sqrt(2) times it is no
// less than the modulus
__device__ __forceinline__ int mag(I2 v) { return max(mag(v.x), mag(v.y)); }

// high word, with and without the bias, of a double that is v 2^e rounded up
__device__ __forceinline__ int high_word(unsigned v, int e) {
  return (__float_as_int(__uint2float_ru(v)) >> 3) + ((1023 - 127 + e) << 20);
}
// Magnitudes of a pencil in fixed point, for the scale of the transform that
// follows: the largest |high word| and their sum, taken in units of 2^39 a value
// and 2^47 a thread, rounded up.
struct FixedNorm {
  unsigned top = 0, sum = 0;
  __device__ __forceinline__ void add(long long v) {
    const unsigned h = unsigned(int(v >> 32) ^ int(v >> 63));
    top = max(top, h);
    sum += (h >> 7) + 1;
  }
  __device__ __forceinline__ unsigned thread_sum() const { return (sum >> 8) + 1; }
};
// over a warp, in a fixed order; f < 2^7
__device__ __forceinline__ float warp_sum(float f) {
  return float(int(__reduce_add_sync(0xffffffffu, unsigned(__float2int_ru(f * 524288.f))))) * (1.f / 524288.f);
}

// Back: values times 2^S; where the exponents leave the range of a double, or
// the input was not finite, every value of the pencil is alt (high word).  The
// conversion is the FP64 pipe's, which has nothing else to do in these kernels
// (half a clock a value beside the 3 of the integer pipe; normalised by integer
// instructions the passes took 6 - 8% longer: 384^3 68.8 against 64.0 ms).
struct OutScale {
  int k;     // S as an exponent's high word
  int alt;
  bool use_alt;
};
__device__ __forceinline__ OutScale out_scale(int em, int S) {
  const bool high = em == 2047 || S + 1086 >= 2047;
  return {S << 20, high ? 0x7ff80000 : 0, high || S + 1086 - 63 <= 0};
}
__device__ __forceinline__ double to_double_p(long long v, const OutScale &o) {
  const double d = __ll2double_rn(v);
  int hi = __double2hiint(d) + o.k;
  hi = v == 0 ? 0 : hi;
  hi = o.use_alt ? o.alt : hi;
  return __hiloint2double(hi, __double2loint(d));
}

// REV: the radices backwards
template <int L, bool REV> struct Fft {
  using D = Len<L>;
  static constexpr int P = 8, lgP = 3, T = D::T, steps = D::steps, W = T / 32;
  static FX_HD constexpr int R(int q) { return D::R(REV ? steps - 1 - q : q); }
  static FX_HD constexpr int NS(int q) { return q == 0 ? 1 : NS(q - 1) * R(q - 1); }
  // butterflies of step q a thread holds
  static FX_HD constexpr int MU(int q) { return (P * (L / R(q)) + T - 1) / T; }
  static constexpr int last = D::steps - 1, lost = bits_lost(last, steps);
  // pencils, then a maximum and a sum of each warp and pencil, twice (k_fx_trunc),
  // or of each of the 16 rows
  static constexpr int norms = W * P * 16 > 128 ? W * P * 16 : 128;
  static constexpr int smem = L * P * 16 + norms;
  // scale of a pencil (fx64.cuh)
  template <FxKind KIND> static __device__ __forceinline__ int scale(int top, int sum) {
    return pencil_scale(top, sum, steps, [](int q) {
      constexpr int lg[3] = {growth(R(0), KIND), growth(R(0) * R(1), KIND), growth(L, KIND)};
      return lg[q];
    });
  }

  static __device__ __forceinline__ int slot(int e, int pen) { return (e << lgP) + (pen ^ (e & (P - 1))); }

  template <int Q> struct Regs {
    I2 v[MU(Q)][R(Q)];
  };
  template <int Q> static __device__ __forceinline__ bool live(int m) {
    constexpr int items = P * (L / R(Q));
    return items % T == 0 || int(threadIdx.x) + m * T < items;
  }
  template <int Q> static __device__ __forceinline__ int jof(int m) { return (int(threadIdx.x) + m * T) >> lgP; }
  // element of input r / output r of butterfly j
  template <int Q> static __device__ __forceinline__ int in_of(int j, int r) { return j + r * (L / R(Q)); }
  template <int Q> static __device__ __forceinline__ int out_of(int j, int r) {
    constexpr int ns = NS(Q);
    return (j / ns) * (ns * R(Q)) + j % ns + r * ns;
  }
  template <int Q> static __device__ __forceinline__ void load(Regs<Q> &g, const longlong2 *s, int pen) {
#pragma unroll
    for (int m = 0; m < MU(Q); ++m)
      if (live<Q>(m)) {
        const int j = jof<Q>(m);
#pragma unroll
        for (int r = 0; r < R(Q); ++r) {
          const longlong2 w = s[slot(in_of<Q>(j, r), pen)];
          g.v[m][r] = {w.x, w.y};
        }
      }
  }
  // FROM, TO: outputs r of FROM < r < TO (both exclusive) are left out
  template <int Q, int FROM = 0, int TO = 0>
  static __device__ __forceinline__ void store(const Regs<Q> &g, longlong2 *s, int pen) {
#pragma unroll
    for (int m = 0; m < MU(Q); ++m)
      if (live<Q>(m)) {
        const int j = jof<Q>(m);
#pragma unroll
        for (int r = 0; r < R(Q); ++r)
          if (!(r > FROM && r < TO)) s[slot(out_of<Q>(j, r), pen)] = make_longlong2(g.v[m][r].x, g.v[m][r].y);
      }
  }
  template <int Q> static __device__ __forceinline__ void butterfly(Regs<Q> &g, const Tw3 &tw) {
    constexpr int ns = NS(Q);
#pragma unroll
    for (int m = 0; m < MU(Q); ++m)
      if (live<Q>(m)) {
        if constexpr (Q > 0) {
          const int inc = (jof<Q>(m) % ns) * (L / (ns * R(Q)));
          if constexpr (doubled(Q, steps)) {
#pragma unroll
            for (int r = 0; r < R(Q); ++r) g.v[m][r] = g.v[m][r] + g.v[m][r];
          }
          g.v[m][0] = quarter(g.v[m][0]);
#pragma unroll
          for (int r = 1; r < R(Q); ++r) g.v[m][r] = twiddle4(g.v[m][r], tw, r * inc);
        }
        Dft<R(Q)>::run(g.v[m]);
      }
  }
  // steps Q .. last, the last one's outputs left to `out` in registers
  template <int Q, class F> static __device__ __forceinline__ void rest(longlong2 *s, int pen, const Tw3 &tw, F &&out) {
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
  // Maximum and sum over the CTA per pencil (lanes of equal low three bits): a
  // warp's four lanes of a pencil first, then the warps, split among these lanes
  // again.  The order is fixed: the scale that comes of it is the same every run.
  static __device__ __forceinline__ int lanes_max(int v) {
    v = max(v, __shfl_xor_sync(0xffffffffu, v, 8));
    return max(v, __shfl_xor_sync(0xffffffffu, v, 16));
  }
  template <class S> static __device__ __forceinline__ S lanes_sum(S v) {
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v + __shfl_xor_sync(0xffffffffu, v, 16);
  }
  static __device__ __forceinline__ float rebase(float f, int top, int to) { return sum_rebase(f, top, to); }
  static __device__ __forceinline__ unsigned rebase(unsigned f, int, int) { return f; }
  template <class S> static __device__ __forceinline__ void pencil_norm(int &top, S &sum, int *wm) {
    const int t = threadIdx.x;
    S *ws = reinterpret_cast<S *>(wm + W * P);
    int own = top;
    top = lanes_max(own);
    sum = lanes_sum(rebase(sum, own, top));
    if constexpr (W > 1) {
      if ((t & 31) < 8) {
        wm[(t >> 5) * 8 + (t & 7)] = top;
        ws[(t >> 5) * 8 + (t & 7)] = sum;
      }
      __syncthreads();
      constexpr int N = (W + 3) / 4;
      int wt[N];
      own = 0;
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const int w = 4 * q + ((t >> 3) & 3);
        wt[q] = W % 4 == 0 || w < W ? wm[w * 8 + (t & 7)] : 0;
        own = max(own, wt[q]);
      }
      top = lanes_max(own);
      sum = 0;
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const int w = 4 * q + ((t >> 3) & 3);
        if (W % 4 == 0 || w < W) sum += rebase(ws[w * 8 + (t & 7)], wt[q], top);
      }
      sum = lanes_sum(sum);
    }
  }
  // scale of the strided passes' pencils from the inputs r that `take` names, and
  // the exponent of their largest component
  template <class G, class T> static __device__ __forceinline__ int norm_scale(const G &g, longlong2 *sm, int &em, T &&take) {
    em = 0;
#pragma unroll
    for (int m = 0; m < MU(0); ++m)
      if (live<0>(m)) {
#pragma unroll
        for (int r = 0; r < R(0); ++r)
          if (take(r)) em = max(em, mag(g.v[m][r]));
      }
    const int base = sum_base(em);
    float sum = 0.f;
#pragma unroll
    for (int m = 0; m < MU(0); ++m)
      if (live<0>(m)) {
#pragma unroll
        for (int r = 0; r < R(0); ++r)
          if (take(r)) sum += sum_term(mag(g.v[m][r]), base);
      }
    pencil_norm(em, sum, norm_at(sm));
    const int k = scale<FX_STRIDED>(em, sum_word(sum, em) + kSqrt2);
    em >>= 20;
    return k;
  }
  // where the norms lie: [warp][pencil], the z passes' [row]
  static __device__ __forceinline__ int *norm_at(longlong2 *sm) { return reinterpret_cast<int *>(sm + L * P); }
  static __device__ __forceinline__ float *row_sums(longlong2 *sm) { return reinterpret_cast<float *>(norm_at(sm) + 2 * P); }
  // scale of the pencil of rows 2 p and 2 p + 1
  template <FxKind KIND> static __device__ __forceinline__ int row_scale(longlong2 *sm, int p, int shift, int &em) {
    const int t0 = norm_at(sm)[2 * p], t1 = norm_at(sm)[2 * p + 1], top = max(t0, t1);
    const float sum = sum_rebase(row_sums(sm)[2 * p], t0, top) + sum_rebase(row_sums(sm)[2 * p + 1], t1, top);
    em = top >> 20;
    return scale<KIND>(top, sum_word(sum, top) + shift);
  }
};

// Where output or input r of the N-grid-side step of a padded length lies:
// rows below N/2, the Nyquist row (butterfly 0 only), the padding, the first
// row above it (not for butterfly 0, which is the padding's last), rows above
enum Zone { Z_LOW, Z_NYQ, Z_PAD, Z_EDGE, Z_HIGH };
template <int R> FX_HD constexpr Zone zone(int r) {
  return r < R / 3 ? Z_LOW : (r == R / 3 ? Z_NYQ : (r < 2 * R / 3 ? Z_PAD : (r == 2 * R / 3 ? Z_EDGE : Z_HIGH)));
}

struct LArgs {
  const void *tw;
  Strided s;
};
struct LRows {
  const void *tw;
  Rows r;
};

// inverse transform along x or y; PAD: N rows in, placed at the padded positions
template <int L, bool PAD>
__global__ void __launch_bounds__(Len<L>::T, Len<L>::ctas) k_fx_inv(const __grid_constant__ LArgs a) {
  mfx::pdl_begin();
  using F = Fft<L, true>;
  extern __shared__ __align__(16) longlong2 sm[];
  const Strided &d = a.s;
  constexpr int R0 = F::R(0), nb = L / R0, nh = L / 3, n = 2 * nh;
  const int t = threadIdx.x, pen = t & 7;
  const Tw3 tw = tw3_of(a.tw, L);
  const int kblocks = (d.kc + 7) >> 3;
  const int o = blockIdx.x / kblocks, kz = ((blockIdx.x - o * kblocks) << 3) + pen;
  const bool lv = kz < d.kc;
  for (int op = d.first[blockIdx.y]; op < d.first[blockIdx.y + 1]; ++op) {
    const double2 *src = static_cast<const double2 *>(d.src[op]) + (long long)o * d.in_outer + kz;
    typename F::template Regs<0> g;
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
        const int j = F::template jof<0>(m);
        const double2 *p = src + (long long)j * d.in_row;
        const long long stride = (long long)nb * d.in_row, back = PAD ? (long long)nh * d.in_row : 0;
#pragma unroll
        for (int r = 0; r < R0; ++r) {
          const Zone z = PAD ? zone<R0>(r) : Z_LOW;
          g.v[m][r] = {0, 0};
          if (z == Z_PAD) continue;
          if (lv && (z == Z_NYQ ? j == 0 : (z == Z_EDGE ? j > 0 : true))) {
            const double2 v = *(p + r * stride - (z >= Z_EDGE ? back : 0));
            g.v[m][r] = {__double_as_longlong(v.x), __double_as_longlong(v.y)};
          }
        }
      }
    if (PAD && (d.pr[op] | d.pk[op]) != 0) {
      const int pr = d.pr[op], pk = d.pk[op];
      const double kk = kz == nh ? 0.0 : double(kz), kf = pk == 2 ? kk * kk : kk;
      const double *mode = d.mode + (pr == 2 ? n : 0);
#pragma unroll
      for (int m = 0; m < F::MU(0); ++m)
        if (F::template live<0>(m)) {
          const int j = F::template jof<0>(m);
#pragma unroll
          for (int r = 0; r < R0; ++r) {
            const Zone z = zone<R0>(r);
            if (z == Z_PAD) continue;
            // padded positions of other butterflies hold zeros: any factor
            const int i = z == Z_NYQ ? nh : j + r * nb - (z >= Z_EDGE ? nh : 0);
            double f = pr ? __ldg(&mode[z == Z_EDGE && j == 0 ? 0 : i]) : kf;
            if (pr && pk) f *= kf;
            g.v[m][r].x = __double_as_longlong(__longlong_as_double(g.v[m][r].x) * f);
            g.v[m][r].y = __double_as_longlong(__longlong_as_double(g.v[m][r].y) * f);
          }
        }
    }
    int em;
    const int k = F::norm_scale(g, sm, em, [](int r) { return !PAD || zone<R0>(r) != Z_PAD; });
    const int sh = shift_of(em, k);
    // inverse transform: real and imaginary part exchanged, here and at the end
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
#pragma unroll
        for (int r = 0; r < R0; ++r)
          if (!PAD || zone<R0>(r) != Z_PAD)
            g.v[m][r] = {to_fixed_p(g.v[m][r].y, sh), to_fixed_p(g.v[m][r].x, sh)};
      }
    F::template butterfly<0>(g, tw);
    F::template store<0>(g, sm, pen);
    __syncthreads();
    const OutScale os = out_scale(em, F::lost - k);
    double2 *dst = static_cast<double2 *>(d.dst[op]) + (long long)o * d.out_outer + kz;
    F::template rest<1>(sm, pen, tw, [&](auto &h) {
      constexpr int Q = F::last;
#pragma unroll
      for (int m = 0; m < F::MU(Q); ++m)
        if (F::template live<Q>(m) && lv) {
          double2 *p = dst + (long long)F::template jof<Q>(m) * d.out_row;
          const long long stride = (long long)F::NS(Q) * d.out_row;
#pragma unroll
          for (int r = 0; r < F::R(Q); ++r)
            p[r * stride] = make_double2(to_double_p(h.v[m][r].y, os), to_double_p(h.v[m][r].x, os));
        }
    });
    if (op + 1 < d.first[blockIdx.y + 1]) __syncthreads();
  }
}

// forward transform along x or y, the N-grid rows kept (the Nyquist row zero);
// inv_lap: times -fac / k^2
template <int L> __global__ void __launch_bounds__(Len<L>::T, Len<L>::ctas) k_fx_cut(const __grid_constant__ LArgs a) {
  mfx::pdl_begin();
  using F = Fft<L, false>;
  extern __shared__ __align__(16) longlong2 sm[];
  const Strided &d = a.s;
  constexpr int R0 = F::R(0), nb = L / R0, nh = L / 3, n = 2 * nh;
  const int t = threadIdx.x, pen = t & 7;
  const Tw3 tw = tw3_of(a.tw, L);
  const int kblocks = (d.kc + 7) >> 3;
  const int o = blockIdx.x / kblocks, kz0 = (blockIdx.x - o * kblocks) << 3, kz = kz0 + pen;
  const bool lv = kz < d.kc;
  const int op = blockIdx.y;
  const double2 *src = static_cast<const double2 *>(d.src[op]) + (long long)o * d.in_outer + kz;
  typename F::template Regs<0> g;
#pragma unroll
  for (int m = 0; m < F::MU(0); ++m)
    if (F::template live<0>(m)) {
      const double2 *p = src + (long long)F::template jof<0>(m) * d.in_row;
      const long long stride = (long long)nb * d.in_row;
#pragma unroll
      for (int r = 0; r < R0; ++r) {
        double2 v = make_double2(0.0, 0.0);
        if (lv) v = p[r * stride];
        g.v[m][r] = {__double_as_longlong(v.x), __double_as_longlong(v.y)};
      }
    }
  int em;
  const int k = F::norm_scale(g, sm, em, [](int) { return true; });
  const int sh = shift_of(em, k);
#pragma unroll
  for (int m = 0; m < F::MU(0); ++m)
    if (F::template live<0>(m)) {
#pragma unroll
      for (int r = 0; r < R0; ++r) g.v[m][r] = {to_fixed_p(g.v[m][r].x, sh), to_fixed_p(g.v[m][r].y, sh)};
    }
  F::template butterfly<0>(g, tw);
  F::template store<0>(g, sm, pen);
  __syncthreads();
  const OutScale os = out_scale(em, F::lost - k);
  double2 *dst = static_cast<double2 *>(d.dst[op]) + (long long)o * d.out_outer + kz;
  F::template rest<1>(sm, pen, tw, [&](auto &h) {
    constexpr int Q = F::last, RL = F::R(Q);
    const bool lap = d.inv_lap;
    const int so = o > nh ? o - n : o, q0 = so * so + kz * kz;
#pragma unroll
    for (int m = 0; m < F::MU(Q); ++m)
      if (F::template live<Q>(m) && lv) {
        const int j = F::template jof<Q>(m);
        double2 *p = dst + (long long)j * d.out_row;
        const long long stride = (long long)F::NS(Q) * d.out_row, back = (long long)nh * d.out_row;
#pragma unroll
        for (int r = 0; r < RL; ++r) {
          const Zone z = zone<RL>(r);
          if (z == Z_PAD || (z == Z_NYQ && j != 0) || (z == Z_EDGE && j == 0)) continue;
          double2 v = make_double2(0.0, 0.0);
          if (z != Z_NYQ) {
            v = make_double2(to_double_p(h.v[m][r].x, os), to_double_p(h.v[m][r].y, os));
            if (lap) {
              const int si = j + r * (L / RL) - (z >= Z_EDGE ? L : 0);  // signed mode index
              const int q = q0 + si * si;
              const double f = o == nh ? 0.0 : -d.fac * __ldg(&d.rinv[q]);  // rinv[0] = 0
              v.x *= f;
              v.y *= f;
            }
          }
          *(p + r * stride - (z >= Z_EDGE ? back : 0)) = v;
        }
      }
  });
  if (d.inv_lap && kz0 + 8 >= d.kc) {
    double2 *z = static_cast<double2 *>(d.dst[op]) + (long long)o * d.out_outer + d.kc;  // the kz Nyquist column
    for (int i = t; i < n; i += F::T) z[(long long)i * d.out_row] = make_double2(0.0, 0.0);
  }
}

// forward, the N-grid rows kept times fac, and back (in place)
template <int L> __global__ void __launch_bounds__(Len<L>::T, Len<L>::ctas) k_fx_trunc(const __grid_constant__ LArgs a) {
  mfx::pdl_begin();
  using F = Fft<L, false>;
  using I = Fft<L, true>;
  extern __shared__ __align__(16) longlong2 sm[];
  const Strided &d = a.s;
  constexpr int R0 = F::R(0), nb = L / R0, RL = F::R(F::last);
  static_assert(F::W > 1, "the second norm's barrier stands before shared memory is written again");
  static_assert(RL == I::R(0), "the forward transform's last radix is the inverse one's first");
  const int t = threadIdx.x, pen = t & 7;
  const Tw3 tw = tw3_of(a.tw, L);
  const int kblocks = (d.kc + 7) >> 3;
  const int o = blockIdx.x / kblocks, kz = ((blockIdx.x - o * kblocks) << 3) + pen;
  const bool lv = kz < d.kc;
  const int op = blockIdx.y;
  typename I::template Regs<0> h;
  int em, k;
  {
    const double2 *src = static_cast<const double2 *>(d.src[op]) + (long long)o * d.in_outer + kz;
    typename F::template Regs<0> g;
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
        const double2 *p = src + (long long)F::template jof<0>(m) * d.in_row;
        const long long stride = (long long)nb * d.in_row;
#pragma unroll
        for (int r = 0; r < R0; ++r) {
          double2 v = make_double2(0.0, 0.0);
          if (lv) v = p[r * stride];
          g.v[m][r] = {__double_as_longlong(v.x), __double_as_longlong(v.y)};
        }
      }
    k = F::norm_scale(g, sm, em, [](int) { return true; });
    const int sh = shift_of(em, k);
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
#pragma unroll
        for (int r = 0; r < R0; ++r) g.v[m][r] = {to_fixed_p(g.v[m][r].x, sh), to_fixed_p(g.v[m][r].y, sh)};
      }
    F::template butterfly<0>(g, tw);
    F::template store<0>(g, sm, pen);
    __syncthreads();
  }
  // the modes outside the N-grid and on its Nyquist row fall away; real and
  // imaginary part are exchanged for the inverse transform
  FixedNorm norm;
  F::template rest<1>(sm, pen, tw, [&](auto &g) {
#pragma unroll
    for (int m = 0; m < F::MU(F::last); ++m)
      if (F::template live<F::last>(m)) {
        const int j = F::template jof<F::last>(m);
#pragma unroll
        for (int r = 0; r < RL; ++r) {
          const Zone z = zone<RL>(r);
          I2 v = g.v[m][r];
          if (z == Z_NYQ || z == Z_PAD || (z == Z_EDGE && j == 0)) v = {0, 0};
          norm.add(v.x);
          norm.add(v.y);
          h.v[m][r] = {v.y, v.x};
        }
      }
  });
  // the scale of the way back, from the high words: a pencil whose values all lie
  // below 2^32 is far below the rounding of the first transform
  int top2 = int(norm.top) + 1;
  unsigned sum2 = norm.thread_sum();
  I::pencil_norm(top2, sum2, I::norm_at(sm) + 2 * F::W * 8);
  const int k2 = I::template scale<FX_STRIDED>(high_word(top2, 32), high_word(sum2, 47) - 0x3ff00000);
  // rescale() without a branch per value
  const int dn = max(-k2, 0), up = max(k2, 0);
  const long long half = dn ? 1LL << (dn - 1) : 0, sign = dn ? -1 : 0;
#pragma unroll
  for (int m = 0; m < I::MU(0); ++m)
    if (I::template live<0>(m)) {
#pragma unroll
      for (int r = 0; r < RL; ++r)
        if (zone<RL>(r) != Z_NYQ && zone<RL>(r) != Z_PAD)
          h.v[m][r] = {((h.v[m][r].x + half + ((h.v[m][r].x >> 63) & sign)) >> dn) << up,
                       ((h.v[m][r].y + half + ((h.v[m][r].y >> 63) & sign)) >> dn) << up};
    }
  I::template butterfly<0>(h, tw);
  I::template store<0>(h, sm, pen);
  __syncthreads();
  const OutScale os = out_scale(em, 2 * F::lost - k - k2);
  double2 *dst = static_cast<double2 *>(d.dst[op]) + (long long)o * d.out_outer + kz;
  I::template rest<1>(sm, pen, tw, [&](auto &g) {
    constexpr int Q = I::last;
#pragma unroll
    for (int m = 0; m < I::MU(Q); ++m)
      if (I::template live<Q>(m) && lv) {
        double2 *p = dst + (long long)I::template jof<Q>(m) * d.out_row;
        const long long stride = (long long)I::NS(Q) * d.out_row;
#pragma unroll
        for (int r = 0; r < I::R(Q); ++r)
          p[r * stride] = make_double2(to_double_p(g.v[m][r].y, os) * d.fac, to_double_p(g.v[m][r].x, os) * d.fac);
      }
  });
}

// spectra -> real rows (fx64.cu k_fx_c2r); PAD: at most L/3 + 1 kz values
template <int L, bool PAD>
__global__ void __launch_bounds__(Len<L>::T, Len<L>::zctas) k_fx_c2r_l(const __grid_constant__ LRows a) {
  mfx::pdl_begin();
  using F = Fft<L, true>;
  extern __shared__ __align__(16) longlong2 sm[];
  const Rows &d = a.r;
  constexpr int h = L / 2, kmax = PAD ? L / 3 + 1 : h, NL = (kmax + 31) / 32;
  const int t = threadIdx.x, lane = t & 31, pen = t & 7;
  const Tw3 tw = tw3_of(a.tw, L);
  double *base = static_cast<double *>(d.field[blockIdx.y]);
  const long long row0 = (long long)blockIdx.x * 16;
  const int kc = min(d.kc, kmax);
  const bool nyq = !PAD && d.kc > h;
#pragma unroll 1
  for (int q = t >> 5; q < 16; q += F::W) {
    const long long row = row0 + q;
    const bool lv = row < d.rows;
    const double2 *src = reinterpret_cast<const double2 *>(base + row * d.pitch);
    const int p = q >> 1, second = q & 1;
    int em = 0;
    double2 v[NL];
#pragma unroll
    for (int c = 0; c < NL; ++c) {
      const int k = lane + 32 * c;
      v[c] = make_double2(0.0, 0.0);
      if (lv && k < kc) v[c] = src[k];
    }
    if (lane == 0) v[0].y = 0.0;  // only the real part of the k = 0 value is used
#pragma unroll
    for (int c = 0; c < NL; ++c) {
      const int k = lane + 32 * c;
      if (k >= (PAD ? kmax : h)) continue;
      const longlong2 b = make_longlong2(__double_as_longlong(v[c].x), __double_as_longlong(v[c].y));
      em = max(em, mag(I2{b.x, b.y}));
      if (k == 0) reinterpret_cast<long long *>(&sm[F::slot(0, p)])[second] = b.x;
      else sm[F::slot(second ? L - k : k, p)] = b;
    }
    int nyq_word = 0;
    if (!PAD && lane == 0) {
      // the Nyquist value (zero where the spectrum ends before it)
      const double x = nyq && lv ? src[h].x : 0.0;
      nyq_word = mag(__double_as_longlong(x));
      em = max(em, nyq_word);
      reinterpret_cast<double *>(&sm[F::slot(h, p)])[second] = x;
    }
    em = int(__reduce_max_sync(0xffffffffu, unsigned(em)));
    const int sb = sum_base(em);
    float sum = sum_term(nyq_word, sb);
#pragma unroll
    for (int c = 0; c < NL; ++c)  // zero beyond the last mode
      sum += sum_term(mag(I2{__double_as_longlong(v[c].x), __double_as_longlong(v[c].y)}), sb);
    sum = warp_sum(sum);
    if (lane == 0) {
      F::norm_at(sm)[q] = em;
      F::row_sums(sm)[q] = sum;
    }
  }
  __syncthreads();
  // every mode but k = 0 and L / 2 stands in the pencil twice
  auto scale_of = [&](int p, int &em) { return F::template row_scale<FX_C2R>(sm, p, kSqrt2 + kTwice, em); };
  {
    int em;
    const int k8 = scale_of(pen, em), sh = shift_of(em, k8);
    auto fix = [&](long long b) { return F::steps > 2 ? to_fixed_r(b, sh) : to_fixed_p(b, sh); };
    constexpr int kend = PAD ? kmax : h;
    for (int k = t >> 3; k < kend; k += F::T / 8) {
      longlong2 &wa = sm[F::slot(k, pen)];
      const longlong2 va = wa;
      const long long ax = fix(va.x), ay = fix(va.y);
      if (k == 0) {
        wa = make_longlong2(ay, ax);
        continue;
      }
      longlong2 &wb = sm[F::slot(L - k, pen)];
      const longlong2 vb = wb;
      const long long bx = fix(vb.x), by = fix(vb.y);
      wa = make_longlong2(ay + bx, ax - by);
      wb = make_longlong2(bx - ay, ax + by);
    }
    if (!PAD && t < 8) {
      longlong2 &w = sm[F::slot(h, t)];
      const longlong2 v = w;
      w = make_longlong2(fix(v.y), fix(v.x));
    }
  }
  __syncthreads();
  {
    // the first step knows the padding (elements L/3 < e < 2L/3) to be zero
    typename F::template Regs<0> g;
    constexpr int R0 = F::R(0);
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
        const int j = F::template jof<0>(m);
#pragma unroll
        for (int r = 0; r < R0; ++r) {
          const Zone z = PAD ? zone<R0>(r) : Z_LOW;
          g.v[m][r] = {0, 0};
          if (z == Z_PAD || (z == Z_NYQ && j != 0)) continue;
          const longlong2 w = sm[F::slot(F::template in_of<0>(j, r), pen)];
          g.v[m][r] = {w.x, w.y};
        }
      }
    F::template butterfly<0>(g, tw);
    __syncthreads();
    F::template store<0>(g, sm, pen);
    __syncthreads();
  }
  F::template rest<1>(sm, pen, tw, [&](auto &g) {
    __syncthreads();
    F::template store<F::last>(g, sm, pen);
    __syncthreads();
  });
#pragma unroll 1
  for (int q = t >> 5; q < 16; q += F::W) {
    const long long row = row0 + q;
    if (row >= d.rows) break;
    double *dst = base + row * d.pitch;
    const int p = q >> 1, second = q & 1;
    int em;
    const int k = scale_of(p, em);
    const OutScale os = out_scale(em, F::lost - k);
#pragma unroll 4
    for (int e = lane; e < L; e += 32)  // exchanged again: the first row is the imaginary part
      dst[e] = to_double_p(reinterpret_cast<const long long *>(&sm[F::slot(e, p)])[1 - second], os);
  }
}

// real rows -> spectra of kz < kc <= L/3 (fx64.cu k_fx_r2c)
template <int L> __global__ void __launch_bounds__(Len<L>::T, Len<L>::zctas) k_fx_r2c_l(const __grid_constant__ LRows a) {
  mfx::pdl_begin();
  using F = Fft<L, false>;
  extern __shared__ __align__(16) longlong2 sm[];
  const Rows &d = a.r;
  constexpr int NL = (L + 31) / 32;
  const int t = threadIdx.x, lane = t & 31, pen = t & 7;
  const Tw3 tw = tw3_of(a.tw, L);
  double *base = static_cast<double *>(d.field[blockIdx.y]);
  const long long row0 = (long long)blockIdx.x * 16;
#pragma unroll 1
  for (int q = t >> 5; q < 16; q += F::W) {
    const long long row = row0 + q;
    const bool lv = row < d.rows;
    const double *src = base + row * d.pitch;
    const int p = q >> 1, second = q & 1;
    int em = 0;
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
        em = max(em, mag(__double_as_longlong(v[c])));
        reinterpret_cast<double *>(&sm[F::slot(e, p)])[second] = v[c];
      }
    }
    em = int(__reduce_max_sync(0xffffffffu, unsigned(em)));
    const int sb = sum_base(em);
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < NL; ++c) sum += sum_term(mag(__double_as_longlong(v[c])), sb);
    sum = warp_sum(sum);
    if (lane == 0) {
      F::norm_at(sm)[q] = em;
      F::row_sums(sm)[q] = sum;
    }
  }
  __syncthreads();
  auto scale_of = [&](int p, int &em) { return F::template row_scale<FX_R2C>(sm, p, 0, em); };
  {
    int em;
    const int k8 = scale_of(pen, em), sh = shift_of(em, k8);
    typename F::template Regs<0> g;
    F::template load<0>(g, sm, pen);
#pragma unroll
    for (int m = 0; m < F::MU(0); ++m)
      if (F::template live<0>(m)) {
#pragma unroll
        for (int r = 0; r < F::R(0); ++r) g.v[m][r] = {to_fixed_p(g.v[m][r].x, sh), to_fixed_p(g.v[m][r].y, sh)};
      }
    F::template butterfly<0>(g, tw);
    __syncthreads();
    F::template store<0>(g, sm, pen);
    __syncthreads();
  }
  F::template rest<1>(sm, pen, tw, [&](auto &g) {
    constexpr int RL = F::R(F::last);
    __syncthreads();
    F::template store<F::last, RL / 3 - 1, 2 * RL / 3>(g, sm, pen);
    __syncthreads();
  });
  const int kc = d.kc;
#pragma unroll 1
  for (int q = t >> 5; q < 16; q += F::W) {
    const long long row = row0 + q;
    if (row >= d.rows) break;
    double2 *dst = reinterpret_cast<double2 *>(base + row * d.pitch);
    const int p = q >> 1, second = q & 1;
    // the sums below are twice the spectra
    int em;
    const int ks = scale_of(p, em);
    const OutScale os = out_scale(em, F::lost - ks - 1);
#pragma unroll 2
    for (int k = lane; k < kc; k += 32) {
      const longlong2 u = sm[F::slot(k, p)], w = sm[F::slot(k ? L - k : 0, p)];
      // A = (Z[k] + conj Z[L-k]) / 2, B = (Z[k] - conj Z[L-k]) / 2i
      const long long x = second ? u.y + w.y : u.x + w.x, y = second ? w.x - u.x : u.y - w.y;
      dst[k] = make_double2(to_double_p(x, os), to_double_p(y, os));
    }
  }
}

// what of a length is launched; a length serves as padded length (multiples of
// three), as grid length, or both
enum FxOp { FX_OP_PREPARE = 0, FX_OP_INV_PAD, FX_OP_CUT, FX_OP_TRUNC, FX_OP_C2R_PAD, FX_OP_R2C, FX_OP_INV, FX_OP_C2R };

// (defined outside the class: an inline member would be instantiated, kernels and
// all, wherever its address is taken)
template <int L, bool PADDED, bool GRID> struct Launch {
  static cudaError_t run(FxOp op, const void *args, dim3 grid, cudaStream_t st);
};
template <int L, bool PADDED, bool GRID>
cudaError_t Launch<L, PADDED, GRID>::run(FxOp op, const void *args, dim3 grid, cudaStream_t st) {
  using F = Fft<L, false>;
  const LArgs *s = static_cast<const LArgs *>(args);
  const LRows *r = static_cast<const LRows *>(args);
  cudaError_t e = cudaSuccess;
  auto limit = [&](const void *f) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, F::smem);
  };
  bool done = op == FX_OP_PREPARE;
  if constexpr (PADDED) {
    if (op == FX_OP_PREPARE) {
      limit((const void *)k_fx_inv<L, true>);
      limit((const void *)k_fx_cut<L>);
      limit((const void *)k_fx_trunc<L>);
      limit((const void *)k_fx_c2r_l<L, true>);
      limit((const void *)k_fx_r2c_l<L>);
    }
    done = true;
    if (op == FX_OP_INV_PAD) mfx::launch_pdl(k_fx_inv<L, true>, grid, F::T, F::smem, st, *s);
    else if (op == FX_OP_CUT) mfx::launch_pdl(k_fx_cut<L>, grid, F::T, F::smem, st, *s);
    else if (op == FX_OP_TRUNC) mfx::launch_pdl(k_fx_trunc<L>, grid, F::T, F::smem, st, *s);
    else if (op == FX_OP_C2R_PAD) mfx::launch_pdl(k_fx_c2r_l<L, true>, grid, F::T, F::smem, st, *r);
    else if (op == FX_OP_R2C) mfx::launch_pdl(k_fx_r2c_l<L>, grid, F::T, F::smem, st, *r);
    else done = op == FX_OP_PREPARE;
  }
  if constexpr (GRID) {
    if (op == FX_OP_PREPARE) {
      limit((const void *)k_fx_inv<L, false>);
      limit((const void *)k_fx_c2r_l<L, false>);
    }
    if (op == FX_OP_INV) {
      mfx::launch_pdl(k_fx_inv<L, false>, grid, F::T, F::smem, st, *s);
      done = true;
    } else if (op == FX_OP_C2R) {
      mfx::launch_pdl(k_fx_c2r_l<L, false>, grid, F::T, F::smem, st, *r);
      done = true;
    }
  }
  if (!done) return cudaErrorInvalidValue;
  return e == cudaSuccess ? cudaGetLastError() : e;
}

}  // namespace fx
