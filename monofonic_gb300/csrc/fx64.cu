// Kernels of the fixed-point transforms (fx64.cuh) of the plain FP64 form and
// their launches.
//
// A 3D transform is three passes over pencils.  A CTA holds P pencils in
// shared memory (16 L P bytes, one buffer: a step reads all its inputs into
// registers before it writes), two steps for most lengths up to 576.
//   load   doubles from HBM into shared memory, largest exponent per pencil
//   steps  Stockham, the first one converting to fixed point as it reads
//   store  back to doubles, to HBM
// Pencils are interleaved ([element][pencil], the pencil index swizzled by the
// element) so that the eight lanes of a 128-byte shared-memory phase always
// read eight different columns, whatever the step's stride.
// Passes skip what the Orszag padding makes zero (the cuFFT route transformed
// it): of the 1.5 M^2 pencils of a padded c2r only N kz/2 + M kz/2 are run
// along y and x, and the Hessian and inverse-Laplacian factors and the
// truncation of convolve3 (convolution.hh:525-532, 552-636) are applied while
// loading and storing.
#include "fx64.cuh"
#include "fx64.h"
#include "fx64_len.cuh"

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

namespace fx {

// for each t < L the three constants of a product with its twiddle, c and s + c
// of all t, then s - c (fx64_len.cuh Tw3)
static void make_twiddles(int L, int4 *cp) {
  int2 *m = reinterpret_cast<int2 *>(cp + L);
  for (int t = 0; t < L; ++t) twiddle_constants(t, L, &cp[t], &m[t]);
}

bool length_supported(int L) { return fx_supported(L); }
const float2 *twiddles32(int L) {
  static std::mutex mu;
  static std::map<int, std::vector<float2>> tables;
  std::lock_guard<std::mutex> lk(mu);
  std::vector<float2> &t = tables[L];
  if (t.empty())
    for (int q = 0; q < L; ++q) {
      const CS w = q62_turn(q, L);
      t.push_back(make_float2(float(std::ldexp(double((long long)w.c), -62)), float(std::ldexp(double((long long)-w.s), -62))));
    }
  return t.data();
}

const void *twiddles(int L) {
  static std::mutex mu;
  static std::map<int, std::vector<int4>> tables;
  std::lock_guard<std::mutex> lk(mu);
  std::vector<int4> &t = tables[L];
  if (t.empty()) {
    t.resize(twiddle_bytes(L) / sizeof(int4));
    make_twiddles(L, t.data());
  }
  return t.data();
}

// ---------------------------------------------------------------------------
// device code
// ---------------------------------------------------------------------------
struct Core {
  FxPlan p;
  const void *tw;
};

__device__ __forceinline__ int slot(int e, int q, int lgP) { return (e << lgP) + (q ^ (e & ((1 << lgP) - 1))); }

// one Stockham step of radix R over the CTA's pencils, a butterfly a thread; raw:
// the values are still doubles (sh: the conversion of this thread's pencil); twice:
// inputs doubled before their twiddles
template <int R>
__device__ __noinline__ void step(const void *tw, int L, int lgP, int NS, unsigned magic, bool raw, int sh, bool twice) {
  extern __shared__ __align__(16) longlong2 s[];
  const int t = threadIdx.x, nb = L / R, pen = t & ((1 << lgP) - 1), j = t >> lgP;
  const bool live = t < (nb << lgP);
  const Tw3 t3 = tw3_of(tw, L);
  I2 v[R];
  int at = 0;
  if (live) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const longlong2 w = s[slot(j + r * nb, pen, lgP)];
      v[r] = {w.x, w.y};
    }
    if (NS == 1) {
      at = j * R;
      if (raw) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = {to_fixed_p(v[r].x, sh), to_fixed_p(v[r].y, sh)};
      }
    } else {
      const int hi = int(__umulhi(unsigned(j), magic)), lo = j - hi * NS, inc = lo * (nb / NS);  // lo L / (NS R)
      at = hi * NS * R + lo;
      if (twice) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = v[r] + v[r];
      }
      v[0] = quarter(v[0]);
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = twiddle4(v[r], t3, r * inc);
    }
    Dft<R>::run(v);
  }
  __syncthreads();
  if (live) {
#pragma unroll
    for (int r = 0; r < R; ++r) s[slot(at + r * NS, pen, lgP)] = make_longlong2(v[r].x, v[r].y);
  }
  __syncthreads();
}

// all steps; ends with a barrier
__device__ __forceinline__ void transform(const Core &c, bool raw, int sh) {
#pragma unroll 1
  for (int q = 0; q < c.p.steps; ++q) {
    const bool rw = raw && q == 0, tw2 = doubled(q, c.p.steps);
    const int L = c.p.L, lgP = c.p.lgP, NS = c.p.NS[q];
    const unsigned mg = c.p.magic[q];
    switch (c.p.R[q]) {
      case 2: step<2>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
      case 3: step<3>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
      case 4: step<4>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
      case 5: step<5>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
      case 6: step<6>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
      case 7: step<7>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
      case 8: step<8>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
      case 9: step<9>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
      case 10: step<10>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
      case 12: step<12>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
      case 14: step<14>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
      case 15: step<15>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
      case 16: step<16>(c.tw, L, lgP, NS, mg, rw, sh, tw2); break;
    }
  }
}

// maximum or sum over the CTA per pencil (threads of equal t mod P), in a fixed
// order; two barriers
template <class S, class F> __device__ __forceinline__ S over_pencil(S v, int P, S *ws, F &&f) {
  const int t = threadIdx.x, pen = t & (P - 1), W = blockDim.x >> 5;
  for (int off = P; off < 32; off <<= 1) v = f(v, __shfl_xor_sync(0xffffffffu, v, off));
  if ((t & 31) < P) ws[(t >> 5) * P + pen] = v;
  __syncthreads();
  v = ws[pen];
  for (int w = 1; w < W; ++w) v = f(v, ws[w * P + pen]);
  __syncthreads();
  return v;
}
struct Max {
  __device__ int operator()(int a, int b) const { return max(a, b); }
};
struct Sum {
  template <class S> __device__ S operator()(S a, S b) const { return a + b; }
};
__device__ __forceinline__ int scale(const Core &c, int top, int sum) {
  return pencil_scale(top, sum, c.p.steps, [&](int q) { return c.p.lg[q]; });
}

// of the pencil of rows 2 p and 2 p + 1
__device__ __forceinline__ int row_scale(const Core &c, const int *rmax, const float *rsum, int p, int shift, int &em) {
  const int t0 = rmax[2 * p], t1 = rmax[2 * p + 1], top = max(t0, t1);
  em = top >> 20;
  return scale(c, top, sum_word(sum_rebase(rsum[2 * p], t0, top) + sum_rebase(rsum[2 * p + 1], t1, top), top) + shift);
}

struct SArgs {
  Core c;
  Strided s;
};

__global__ void __launch_bounds__(768) k_fx_strided(const __grid_constant__ SArgs a) {
  mfx::pdl_begin();
  extern __shared__ __align__(16) longlong2 sm[];
  const Strided &d = a.s;
  const int L = a.c.p.L, lgP = a.c.p.lgP, P = 1 << lgP, T = blockDim.x, t = threadIdx.x;
  void *norm_at = sm + (size_t(L) << lgP);
  const int kblocks = (d.kc + P - 1) >> lgP;
  const int o = blockIdx.x / kblocks, kz0 = (blockIdx.x - o * kblocks) << lgP;
  const int pen = t & (P - 1), kz = kz0 + pen;
  const bool live = kz < d.kc;
  const int n = d.n, nh = n >> 1;
  const int step_l = T >> lgP;
  for (int op = d.first[blockIdx.y]; op < d.first[blockIdx.y + 1]; ++op) {
    // load
    const double2 *src = static_cast<const double2 *>(d.src[op]) + (long long)o * d.in_outer + kz;
    const int pr = d.pr[op], pk = d.pk[op];
    const bool scaled = (pr | pk) != 0;
    const double kf = pk == 0 ? 1.0 : ((d.inverse && kz == nh) ? 0.0 : (pk == 1 ? double(kz) : double(kz) * double(kz)));
    int em = 0;
#pragma unroll 4
    for (int l = t >> lgP; l < L; l += step_l) {
      double2 v = make_double2(0.0, 0.0);
      const int i = !d.pad_in ? l : (l <= nh ? l : (l > n ? l - nh : -1));
      if (live && i >= 0) {
        v = src[(long long)i * d.in_row];
        if (scaled) {
          const double f = (pr ? __ldg(&d.mode[(pr - 1) * n + i]) : 1.0) * kf;
          v.x *= f;
          v.y *= f;
        }
      }
      em = max(em, mag(I2{__double_as_longlong(v.x), __double_as_longlong(v.y)}));
      sm[slot(l, pen, lgP)] = d.inverse ? make_longlong2(__double_as_longlong(v.y), __double_as_longlong(v.x))
                                        : make_longlong2(__double_as_longlong(v.x), __double_as_longlong(v.y));
    }
    em = over_pencil(em, P, static_cast<int *>(norm_at), Max());
    float sum = 0.f;
    for (int l = t >> lgP; l < L; l += step_l) {
      const longlong2 w = sm[slot(l, pen, lgP)];
      sum += sum_term(mag(I2{w.x, w.y}), sum_base(em));
    }
    sum = over_pencil(sum, P, static_cast<float *>(norm_at), Sum());
    const int k = scale(a.c, em, sum_word(sum, em) + kSqrt2);
    em >>= 20;
    const int lost = bits_lost(a.c.p.steps - 1, a.c.p.steps);
    int S = lost - k;
    transform(a.c, true, shift_of(em, k));
    bool inverse = d.inverse;
    if (d.truncate) {
      // keep the N-grid modes, scale for the way back (fx64_len.cuh k_fx_trunc),
      // swap for the inverse transform (inverse = swap, forward, swap)
      FixedNorm norm;
      for (int l = t >> lgP; l < L; l += step_l) {
        const bool keep = l < nh || l > n;
        longlong2 &w = sm[slot(l, pen, lgP)];
        const longlong2 v = w;
        if (keep) {
          norm.add(v.x);
          norm.add(v.y);
        }
        w = keep ? make_longlong2(v.y, v.x) : make_longlong2(0, 0);
      }
      const int top2 = over_pencil(int(norm.top) + 1, P, static_cast<int *>(norm_at), Max());
      const unsigned sum2 = over_pencil(norm.thread_sum(), P, static_cast<unsigned *>(norm_at), Sum());
      const int k2 = scale(a.c, high_word(top2, 32), high_word(sum2, 47) - 0x3ff00000);
      for (int l = t >> lgP; l < L; l += step_l) {
        longlong2 &w = sm[slot(l, pen, lgP)];
        w = make_longlong2(rescale(w.x, k2), rescale(w.y, k2));
      }
      __syncthreads();
      S += lost - k2;
      transform(a.c, false, 0);
      inverse = true;
    }
    // store
    double2 *dst = static_cast<double2 *>(d.dst[op]) + (long long)o * d.out_outer + kz;
    const int so = o > nh ? o - n : o;
    const OutScale os = out_scale(em, S);
    for (int l = t >> lgP; l < L; l += step_l) {
      const int i = !d.cut_out ? l : (l <= nh ? l : (l > n ? l - nh : -1));
      if (i < 0 || !live) continue;
      const longlong2 w = sm[slot(l, pen, lgP)];
      double2 v = make_double2(to_double_p(w.x, os), to_double_p(w.y, os));
      if (inverse) v = make_double2(v.y, v.x);
      if (d.cut_out) {
        if (i == nh || (d.inv_lap && (o == nh || (o | i | kz) == 0))) {
          v = make_double2(0.0, 0.0);
        } else if (d.inv_lap) {
          const int si = i > nh ? i - n : i;
          const double f = -d.fac * __ldg(&d.rinv[so * so + si * si + kz * kz]);
          v.x *= f;
          v.y *= f;
        }
      } else if (d.truncate) {
        v.x *= d.fac;
        v.y *= d.fac;
      }
      dst[(long long)i * d.out_row] = v;
    }
    if (d.inv_lap && kz0 + P >= d.kc) {
      // the kz Nyquist column
      double2 *z = static_cast<double2 *>(d.dst[op]) + (long long)o * d.out_outer + d.kc;
      for (int i = t; i < n; i += T) z[(long long)i * d.out_row] = make_double2(0.0, 0.0);
    }
    __syncthreads();
  }
}

struct RArgs {
  Core c;
  Rows r;
};

// spectra -> real rows: rows 2q and 2q + 1 as the real and imaginary part of
// one pencil, Z[k] = A[k] + i B[k], Z[L - k] = conj A[k] + i conj B[k]
__global__ void __launch_bounds__(768) k_fx_c2r(const __grid_constant__ RArgs a) {
  mfx::pdl_begin();
  extern __shared__ __align__(16) longlong2 sm[];
  const Rows &d = a.r;
  const int L = a.c.p.L, lgP = a.c.p.lgP, P = 1 << lgP, T = blockDim.x, t = threadIdx.x, lane = t & 31;
  int *rmax = reinterpret_cast<int *>(sm + (size_t(L) << lgP));  // per row
  float *rsum = reinterpret_cast<float *>(rmax + 2 * P);
  double *base = static_cast<double *>(d.field[blockIdx.y]);
  const long long row0 = (long long)blockIdx.x * 2 * P;
  const int h = L >> 1, kc = min(d.kc, h);  // the Nyquist value, if any, is handled apart
  const bool nyq = d.kc > h;
  // zero the elements without a mode
  for (int e = t; e < ((L - 2 * kc + 1) << lgP); e += T) sm[slot(kc + (e >> lgP), e & (P - 1), lgP)] = make_longlong2(0, 0);
  __syncthreads();
  for (int q = t >> 5; q < 2 * P; q += T >> 5) {
    const long long row = row0 + q;
    const bool live = row < d.rows;
    const double2 *src = reinterpret_cast<const double2 *>(base + row * d.pitch);
    const int pen = q >> 1, second = q & 1;
    int em = 0;
#pragma unroll 4
    for (int k = lane; k < kc; k += 32) {
      double2 v = live ? src[k] : make_double2(0.0, 0.0);
      if (k == 0) {
        // only the real part of the k = 0 (and the Nyquist) value is used
        em = max(em, mag(__double_as_longlong(v.x)));
        reinterpret_cast<double *>(&sm[slot(0, pen, lgP)])[second] = v.x;
      } else {
        em = max(em, mag(I2{__double_as_longlong(v.x), __double_as_longlong(v.y)}));
        sm[slot(second ? L - k : k, pen, lgP)] = make_longlong2(__double_as_longlong(v.x), __double_as_longlong(v.y));
      }
    }
    int nyq_word = 0;
    if (nyq && lane == 0) {
      const double v = live ? src[h].x : 0.0;
      nyq_word = mag(__double_as_longlong(v));
      em = max(em, nyq_word);
      reinterpret_cast<double *>(&sm[slot(h, pen, lgP)])[second] = v;
    }
    em = __reduce_max_sync(0xffffffffu, unsigned(em));
    const int sb = sum_base(em);
    float sum = sum_term(nyq_word, sb);
    for (int k = lane; k < kc; k += 32) {  // what this lane has just written
      const longlong2 w = sm[slot(second && k ? L - k : k, pen, lgP)];
      sum += sum_term(k ? mag(I2{w.x, w.y}) : mag(second ? w.y : w.x), sb);
    }
    sum = warp_sum(sum);
    if (lane == 0) {
      rmax[q] = em;
      rsum[q] = sum;
    }
  }
  __syncthreads();
  // every mode but k = 0 and L / 2 stands in the pencil twice
  auto scale_of = [&](int p, int &em) { return row_scale(a.c, rmax, rsum, p, kSqrt2 + kTwice, em); };
  {
    // Z of both rows in fixed point, real and imaginary part exchanged (the
    // inverse transform)
    const int pen = t & (P - 1);
    int em;
    const int k8 = scale_of(pen, em), sh = shift_of(em, k8);
    const bool round = a.c.p.steps > 2;
    auto fix = [&](long long b) { return round ? to_fixed_r(b, sh) : to_fixed_p(b, sh); };
    for (int k = t >> lgP; k < kc; k += T >> lgP) {
      longlong2 &wa = sm[slot(k, pen, lgP)];
      const longlong2 va = wa;
      const long long ax = fix(va.x), ay = fix(va.y);
      if (k == 0) {
        wa = make_longlong2(ay, ax);
        continue;
      }
      longlong2 &wb = sm[slot(L - k, pen, lgP)];
      const longlong2 vb = wb;
      const long long bx = fix(vb.x), by = fix(vb.y);
      wa = make_longlong2(ay + bx, ax - by);
      wb = make_longlong2(bx - ay, ax + by);
    }
    if (nyq && t < P) {
      longlong2 &w = sm[slot(h, t, lgP)];
      const longlong2 v = w;
      w = make_longlong2(fix(v.y), fix(v.x));
    }
  }
  __syncthreads();
  transform(a.c, false, 0);
  for (int q = t >> 5; q < 2 * P; q += T >> 5) {
    const long long row = row0 + q;
    if (row >= d.rows) break;
    double *dst = base + row * d.pitch;
    const int pen = q >> 1, second = q & 1;
    int em;
    const int k = scale_of(pen, em);
    const OutScale os = out_scale(em, bits_lost(a.c.p.steps - 1, a.c.p.steps) - k);
    for (int e = lane; e < L; e += 32)  // exchanged again: the first row is the imaginary part
      dst[e] = to_double_p(reinterpret_cast<const long long *>(&sm[slot(e, pen, lgP)])[1 - second], os);
  }
}

// real rows -> spectra of kz < kc, two rows a pencil
__global__ void __launch_bounds__(768) k_fx_r2c(const __grid_constant__ RArgs a) {
  mfx::pdl_begin();
  extern __shared__ __align__(16) longlong2 sm[];
  const Rows &d = a.r;
  const int L = a.c.p.L, lgP = a.c.p.lgP, P = 1 << lgP, T = blockDim.x, t = threadIdx.x, lane = t & 31;
  int *rmax = reinterpret_cast<int *>(sm + (size_t(L) << lgP));  // per row
  float *rsum = reinterpret_cast<float *>(rmax + 2 * P);
  double *base = static_cast<double *>(d.field[blockIdx.y]);
  const long long row0 = (long long)blockIdx.x * 2 * P;
  for (int q = t >> 5; q < 2 * P; q += T >> 5) {
    const long long row = row0 + q;
    const bool live = row < d.rows;
    const double *src = base + row * d.pitch;
    const int pen = q >> 1, second = q & 1;
    int em = 0;
#pragma unroll 8
    for (int e = lane; e < L; e += 32) {
      const double v = live ? src[e] : 0.0;
      em = max(em, mag(__double_as_longlong(v)));
      reinterpret_cast<double *>(&sm[slot(e, pen, lgP)])[second] = v;
    }
    em = __reduce_max_sync(0xffffffffu, unsigned(em));
    const int sb = sum_base(em);
    float sum = 0.f;
    for (int e = lane; e < L; e += 32)  // what this lane has just written
      sum += sum_term(mag(reinterpret_cast<const long long *>(&sm[slot(e, pen, lgP)])[second]), sb);
    sum = warp_sum(sum);
    if (lane == 0) {
      rmax[q] = em;
      rsum[q] = sum;
    }
  }
  __syncthreads();
  auto scale_of = [&](int p, int &em) { return row_scale(a.c, rmax, rsum, p, 0, em); };
  {
    int em;
    const int k = scale_of(t & (P - 1), em);
    transform(a.c, true, shift_of(em, k));
  }
  const int kc = d.kc;
  for (int q = t >> 5; q < 2 * P; q += T >> 5) {
    const long long row = row0 + q;
    if (row >= d.rows) break;
    double2 *dst = reinterpret_cast<double2 *>(base + row * d.pitch);
    const int pen = q >> 1, second = q & 1;
    // the sums below are twice the spectra
    int em;
    const int ks = scale_of(pen, em);
    const OutScale os = out_scale(em, bits_lost(a.c.p.steps - 1, a.c.p.steps) - ks - 1);
    for (int k = lane; k < kc; k += 32) {
      const longlong2 u = sm[slot(k, pen, lgP)], w = sm[slot(k ? L - k : 0, pen, lgP)];
      // A = (Z[k] + conj Z[L-k]) / 2, B = (Z[k] - conj Z[L-k]) / 2i
      const long long x = second ? u.y + w.y : u.x + w.x, y = second ? w.x - u.x : u.y - w.y;
      dst[k] = make_double2(to_double_p(x, os), to_double_p(y, os));
    }
  }
}

// ---------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------
// the instance of a length, if it has one: as padded length, as grid length
using LenFn = cudaError_t (*)(FxOp, const void *, dim3, cudaStream_t);
struct LenEntry {
  int L;
  bool padded, grid;
  LenFn fn;
};
#define FX_EXTERN(L, PADDED, GRID) extern template struct Launch<L, PADDED, GRID>;
FX_LENGTHS(FX_EXTERN)
#define FX_ENTRY(L, PADDED, GRID) {L, PADDED, GRID, Launch<L, PADDED, GRID>::run},
static const LenEntry kLens[] = {FX_LENGTHS(FX_ENTRY)};
static const LenEntry *find_len(int L) {
  for (const LenEntry &e : kLens)
    if (e.L == L) return &e;
  return nullptr;
}
static __global__ void k_fx_tables(int n, double *mode, double *rinv, double *root, int len) {
  mfx::pdl_begin();
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < len; q += gridDim.x * blockDim.x) {
    rinv[q] = q ? 1.0 / double(q) : 0.0;
    root[q] = sqrt(double(q));
    if (q < n) {
      const int i = q == n / 2 ? 0 : (q > n / 2 ? q - n : q);
      mode[q] = double(i);
      mode[n + q] = double(i) * double(i);
      const double ratio = 64.0 / double(n), x = double(q) * ratio, f = floor(x);
      mode[2 * n + q] = x - f;
      mode[3 * n + q] = (x - (x > 32.0 ? 64.0 : 0.0)) / ratio;
      reinterpret_cast<int *>(mode + 4 * n)[q] = int(f);
    }
  }
}
cudaError_t fill_tables(int n, double *mode, double *rinv, double *root, cudaStream_t st) {
  const int len = int(rinv_len(n));
  mfx::launch_pdl(k_fx_tables, unsigned(std::min((len + 255) / 256, 608)), 256, 0, st, n, mode, rinv, root, len);
  return cudaGetLastError();
}

cudaError_t prepare_device(int dev) {
  static std::mutex mu;
  static std::vector<bool> done;
  std::lock_guard<std::mutex> lk(mu);
  if (dev < int(done.size()) && done[dev]) return cudaSuccess;
  for (const void *f : {(const void *)k_fx_strided, (const void *)k_fx_c2r, (const void *)k_fx_r2c}) {
    const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    if (e != cudaSuccess) return e;
  }
  for (const LenEntry &l : kLens) {
    const cudaError_t e = l.fn(FX_OP_PREPARE, nullptr, dim3(), nullptr);
    if (e != cudaSuccess) return e;
  }
  if (dev >= int(done.size())) done.resize(dev + 1, false);
  done[dev] = true;
  return cudaSuccess;
}

cudaError_t run_strided(const Strided &s, cudaStream_t st) {
  if (const LenEntry *l = find_len(s.L)) {
    const bool p = l->padded && 3 * s.n == 2 * s.L;
    const bool single = s.groups == s.ops;
    FxOp op = FX_OP_PREPARE;
    if (s.inverse && !s.cut_out && !s.truncate) op = s.pad_in ? (p ? FX_OP_INV_PAD : op) : (l->grid ? FX_OP_INV : op);
    else if (!s.inverse && !s.pad_in && single) op = !p ? op : (s.truncate ? FX_OP_TRUNC : (s.cut_out ? FX_OP_CUT : op));
    if (op != FX_OP_PREPARE) {
      const LArgs a{s.tw, s};
      return l->fn(op, &a, dim3(unsigned(s.outer * ((s.kc + 7) / 8)), unsigned(s.groups)), st);
    }
  }
  SArgs a;
  if (!fx_plan(s.L, FX_STRIDED, &a.c.p)) return cudaErrorInvalidValue;
  a.c.tw = s.tw;
  a.s = s;
  const int kb = (s.kc + a.c.p.P - 1) / a.c.p.P;
  mfx::launch_pdl(k_fx_strided, dim3(unsigned(s.outer * kb), unsigned(s.groups)), a.c.p.T, a.c.p.smem, st, a);
  return cudaGetLastError();
}

static cudaError_t run_rows(const Rows &r, FxKind kind, cudaStream_t st) {
  if (const LenEntry *l = find_len(r.L)) {
    FxOp op = FX_OP_PREPARE;
    if (kind == FX_C2R) op = l->padded && r.kc <= r.L / 3 + 1 ? FX_OP_C2R_PAD : (l->grid ? FX_OP_C2R : op);
    else if (l->padded && r.kc <= r.L / 3) op = FX_OP_R2C;
    if (op != FX_OP_PREPARE) {
      const LRows a{r.tw, r};
      return l->fn(op, &a, dim3(unsigned((r.rows + 15) / 16), unsigned(r.count)), st);
    }
  }
  RArgs a;
  if (!fx_plan(r.L, kind, &a.c.p)) return cudaErrorInvalidValue;
  a.c.tw = r.tw;
  a.r = r;
  const long long per = 2 * a.c.p.P;
  const dim3 grid(unsigned((r.rows + per - 1) / per), unsigned(r.count));
  if (kind == FX_C2R) mfx::launch_pdl(k_fx_c2r, grid, a.c.p.T, a.c.p.smem, st, a);
  else mfx::launch_pdl(k_fx_r2c, grid, a.c.p.T, a.c.p.smem, st, a);
  return cudaGetLastError();
}
cudaError_t run_c2r(const Rows &r, cudaStream_t st) { return run_rows(r, FX_C2R, st); }
cudaError_t run_r2c(const Rows &r, cudaStream_t st) { return run_rows(r, FX_R2C, st); }

}  // namespace fx
