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

// ---------------------------------------------------------------------------
// plans
// ---------------------------------------------------------------------------
namespace {
constexpr int kRadices[] = {16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
constexpr int kSmemMax = 220 * 1024;

// rough cost of a point: real multiplications (three products each, measured
// 4 a clock) and the shared-memory round trip of a step
double radix_cost(int R) {
  switch (R) {
    case 2: case 4: return 0.0;
    case 3: return 0.67; case 5: return 2.0; case 6: return 0.67; case 7: return 5.1;
    case 8: return 0.5; case 9: return 2.0; case 10: return 2.0; case 12: return 0.67;
    case 14: return 5.1; case 15: return 2.67; default: return 1.25;  // 16
  }
}

// best factorisation: fewest steps, then least cost, then smallest largest radix
void search(int rest, int depth, double cost, int *cur, int &best_n, double &best_c, int *best) {
  if (rest == 1) {
    int mx = 0;
    for (int q = 0; q < depth; ++q) mx = std::max(mx, cur[q]);
    const double c = cost + 0.02 * mx;
    if (depth < best_n || (depth == best_n && c < best_c)) {
      best_n = depth;
      best_c = c;
      std::copy(cur, cur + depth, best);
    }
    return;
  }
  if (depth == kMaxSteps || depth >= best_n) return;
  for (int R : kRadices)
    if (rest % R == 0 && (depth == 0 || R <= cur[depth - 1])) {
      cur[depth] = R;
      search(rest / R, depth + 1, cost + radix_cost(R), cur, best_n, best_c, best);
    }
}
}  // namespace

int fx_bits(const int *R, int steps, FxKind kind) {
  double m = kind == FX_C2R ? 1.5 : 0.5, top = m;
  for (int q = 0; q < steps; ++q) {
    if (q) m -= 3.0;
    m += std::log2(double(R[q]));
    top = std::max(top, m);
  }
  if (kind == FX_R2C) top = std::max(top, m + 1.0);
  return std::min(60, int(std::floor(62.7 - top)));
}

bool fx_plan(int L, FxKind kind, FxPlan *p) {
  *p = FxPlan{};
  p->L = L;
  int cur[kMaxSteps], best[kMaxSteps], n = kMaxSteps + 1;
  double c = 1e30;
  search(L, 0, 0.0, cur, n, c, best);
  if (n > kMaxSteps) return false;
  p->steps = n;
  // smallest radix first: its butterflies, the most, carry no twiddles
  std::sort(best, best + n);
  int ns = 1;
  for (int q = 0; q < n; ++q) {
    p->R[q] = best[q];
    p->NS[q] = ns;
    p->magic[q] = unsigned((0x100000000ULL + unsigned(ns) - 1) / unsigned(ns));
    ns *= best[q];
  }
  p->B = fx_bits(p->R, n, kind);
  for (int P : {8, 4, 2, 1}) {
    int need = 32;  // threads: a butterfly each
    for (int q = 0; q < n; ++q) need = std::max(need, P * (L / p->R[q]));
    const int T = (need + 31) / 32 * 32;
    const int smem = L * P * 16 + P * 8;
    if (T > 768 || smem > kSmemMax) continue;
    p->P = P;
    p->lgP = P == 8 ? 3 : (P == 4 ? 2 : P - 1);
    p->T = T;
    p->smem = smem;
    return true;
  }
  return false;
}

// (cos, -sin)(2 pi t / L) 2^61, t < L, then the three constants of the products
// with them, split into signed halves: c and s + c, then s - c (fx64_len.cuh Tw3)
static void make_twiddles(int L, longlong2 *out) {
  int4 *cp = reinterpret_cast<int4 *>(out + L);
  int2 *m = reinterpret_cast<int2 *>(cp + L);
  auto lo = [](long long w) { return int(w); };
  auto hi = [](long long w) { return int(w >> 32) + int(unsigned(int(w)) >> 31); };
  for (int t = 0; t < L; ++t) {
    const CS w = q62_turn(t, L);
    const long long c = (long long)((w.c + 1) >> 1), s = (long long)((-w.s + 1) >> 1);
    out[t] = make_longlong2(c, s);
    cp[t] = make_int4(hi(c), lo(c), hi(s + c), lo(s + c));
    m[t] = make_int2(hi(s - c), lo(s - c));
  }
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

const longlong2 *twiddles(int L) {
  static std::mutex mu;
  static std::map<int, std::vector<longlong2>> tables;
  std::lock_guard<std::mutex> lk(mu);
  std::vector<longlong2> &t = tables[L];
  if (t.empty()) {
    t.resize(twiddle_bytes(L) / sizeof(longlong2));
    make_twiddles(L, t.data());
  }
  return t.data();
}

// ---------------------------------------------------------------------------
// device code
// ---------------------------------------------------------------------------
struct Core {
  FxPlan p;
  const longlong2 *tw;
};

__device__ __forceinline__ int slot(int e, int q, int lgP) { return (e << lgP) + (q ^ (e & ((1 << lgP) - 1))); }

// one Stockham step of radix R over the CTA's pencils, a butterfly a thread; raw:
// the values are still doubles (sh: the conversion of this thread's pencil)
template <int R>
__device__ __noinline__ void step(const longlong2 *tw, int L, int lgP, int NS, unsigned magic, bool raw, int sh) {
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
      v[0] = eighth(v[0]);
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = twiddle8(v[r], t3, r * inc);
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
    const bool rw = raw && q == 0;
    const int L = c.p.L, lgP = c.p.lgP, NS = c.p.NS[q];
    const unsigned mg = c.p.magic[q];
    switch (c.p.R[q]) {
      case 2: step<2>(c.tw, L, lgP, NS, mg, rw, sh); break;
      case 3: step<3>(c.tw, L, lgP, NS, mg, rw, sh); break;
      case 4: step<4>(c.tw, L, lgP, NS, mg, rw, sh); break;
      case 5: step<5>(c.tw, L, lgP, NS, mg, rw, sh); break;
      case 6: step<6>(c.tw, L, lgP, NS, mg, rw, sh); break;
      case 7: step<7>(c.tw, L, lgP, NS, mg, rw, sh); break;
      case 8: step<8>(c.tw, L, lgP, NS, mg, rw, sh); break;
      case 9: step<9>(c.tw, L, lgP, NS, mg, rw, sh); break;
      case 10: step<10>(c.tw, L, lgP, NS, mg, rw, sh); break;
      case 12: step<12>(c.tw, L, lgP, NS, mg, rw, sh); break;
      case 14: step<14>(c.tw, L, lgP, NS, mg, rw, sh); break;
      case 15: step<15>(c.tw, L, lgP, NS, mg, rw, sh); break;
      case 16: step<16>(c.tw, L, lgP, NS, mg, rw, sh); break;
    }
  }
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
  int *emax = reinterpret_cast<int *>(sm + (size_t(L) << lgP));
  const int kblocks = (d.kc + P - 1) >> lgP;
  const int o = blockIdx.x / kblocks, kz0 = (blockIdx.x - o * kblocks) << lgP;
  const int pen = t & (P - 1), kz = kz0 + pen;
  const bool live = kz < d.kc;
  const int n = d.n, nh = n >> 1;
  const int step_l = T >> lgP;
  for (int op = d.first[blockIdx.y]; op < d.first[blockIdx.y + 1]; ++op) {
    if (t < P) emax[t] = 0;
    __syncthreads();
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
      em = max(em, max(mag(__double_as_longlong(v.x)), mag(__double_as_longlong(v.y))));
      sm[slot(l, pen, lgP)] = d.inverse ? make_longlong2(__double_as_longlong(v.y), __double_as_longlong(v.x))
                                        : make_longlong2(__double_as_longlong(v.x), __double_as_longlong(v.y));
    }
    for (int off = P; off < 32; off <<= 1) em = max(em, __shfl_xor_sync(0xffffffffu, em, off));
    if ((t & 31) < P) atomicMax(&emax[pen], em);
    __syncthreads();
    em = emax[pen] >> 20;
    int S = em - 1022 - a.c.p.B + 3 * (a.c.p.steps - 1);
    transform(a.c, true, shift_of(em, a.c.p.B));
    bool inverse = d.inverse;
    if (d.truncate) {
      // keep the N-grid modes, bring the largest back below 2^B, swap for the
      // inverse transform (inverse = swap, forward, swap)
      int bits = 0;
      for (int l = t >> lgP; l < L; l += step_l) {
        const bool keep = l < nh || l > n;
        longlong2 &w = sm[slot(l, pen, lgP)];
        const longlong2 v = w;
        if (keep) bits = max(bits, 64 - min(__clzll(v.x ^ (v.x >> 63)), __clzll(v.y ^ (v.y >> 63))));
        w = keep ? make_longlong2(v.y, v.x) : make_longlong2(0, 0);
      }
      if (t < P) emax[t] = 0;
      __syncthreads();
      for (int off = P; off < 32; off <<= 1) bits = max(bits, __shfl_xor_sync(0xffffffffu, bits, off));
      if ((t & 31) < P) atomicMax(&emax[pen], bits);
      __syncthreads();
      const int down = emax[pen] - a.c.p.B;
      for (int l = t >> lgP; l < L; l += step_l) {
        longlong2 &w = sm[slot(l, pen, lgP)];
        if (down > 0) {
          const long long half = 1LL << (down - 1);
          w = make_longlong2((w.x + half) >> down, (w.y + half) >> down);
        } else {
          w = make_longlong2(w.x << -down, w.y << -down);
        }
      }
      __syncthreads();
      S += down + 3 * (a.c.p.steps - 1);
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
  int *emax = reinterpret_cast<int *>(sm + (size_t(L) << lgP));
  double *base = static_cast<double *>(d.field[blockIdx.y]);
  const long long row0 = (long long)blockIdx.x * 2 * P;
  const int h = L >> 1, kc = min(d.kc, h);  // the Nyquist value, if any, is handled apart
  const bool nyq = d.kc > h;
  if (t < P) emax[t] = 0;
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
        em = max(em, max(mag(__double_as_longlong(v.x)), mag(__double_as_longlong(v.y))));
        sm[slot(second ? L - k : k, pen, lgP)] = make_longlong2(__double_as_longlong(v.x), __double_as_longlong(v.y));
      }
    }
    if (nyq && lane == 0) {
      const double v = live ? src[h].x : 0.0;
      em = max(em, mag(__double_as_longlong(v)));
      reinterpret_cast<double *>(&sm[slot(h, pen, lgP)])[second] = v;
    }
    em = __reduce_max_sync(0xffffffffu, unsigned(em));
    if (lane == 0) atomicMax(&emax[pen], em);
  }
  __syncthreads();
  {
    // Z of both rows in fixed point, real and imaginary part exchanged (the
    // inverse transform)
    const int pen = t & (P - 1), sh = shift_of(emax[pen] >> 20, a.c.p.B);
    for (int k = t >> lgP; k < kc; k += T >> lgP) {
      longlong2 &wa = sm[slot(k, pen, lgP)];
      const longlong2 va = wa;
      const long long ax = to_fixed_p(va.x, sh), ay = to_fixed_p(va.y, sh);
      if (k == 0) {
        wa = make_longlong2(ay, ax);
        continue;
      }
      longlong2 &wb = sm[slot(L - k, pen, lgP)];
      const longlong2 vb = wb;
      const long long bx = to_fixed_p(vb.x, sh), by = to_fixed_p(vb.y, sh);
      wa = make_longlong2(ay + bx, ax - by);
      wb = make_longlong2(bx - ay, ax + by);
    }
    if (nyq && t < P) {
      longlong2 &w = sm[slot(h, t, lgP)];
      const longlong2 v = w;
      w = make_longlong2(to_fixed_p(v.y, sh), to_fixed_p(v.x, sh));
    }
  }
  __syncthreads();
  transform(a.c, false, 0);
  for (int q = t >> 5; q < 2 * P; q += T >> 5) {
    const long long row = row0 + q;
    if (row >= d.rows) break;
    double *dst = base + row * d.pitch;
    const int pen = q >> 1, second = q & 1;
    const int em = emax[pen] >> 20;
    const OutScale os = out_scale(em, em - 1022 - a.c.p.B + 3 * (a.c.p.steps - 1));
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
  int *emax = reinterpret_cast<int *>(sm + (size_t(L) << lgP));
  double *base = static_cast<double *>(d.field[blockIdx.y]);
  const long long row0 = (long long)blockIdx.x * 2 * P;
  if (t < P) emax[t] = 0;
  __syncthreads();
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
    if (lane == 0) atomicMax(&emax[pen], em);
  }
  __syncthreads();
  transform(a.c, true, shift_of(emax[t & (P - 1)] >> 20, a.c.p.B));
  const int kc = d.kc;
  for (int q = t >> 5; q < 2 * P; q += T >> 5) {
    const long long row = row0 + q;
    if (row >= d.rows) break;
    double2 *dst = reinterpret_cast<double2 *>(base + row * d.pitch);
    const int pen = q >> 1, second = q & 1;
    // the sums below are twice the spectra
    const int em = emax[pen] >> 20;
    const OutScale os = out_scale(em, em - 1022 - a.c.p.B + 3 * (a.c.p.steps - 1) - 1);
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
  int steps, R[3];  // in the order of a forward transform
};
extern template struct Launch<16, false, true>;
extern template struct Launch<24, true, true>;
extern template struct Launch<32, false, true>;
extern template struct Launch<48, true, true>;
extern template struct Launch<64, false, true>;
extern template struct Launch<72, true, true>;
extern template struct Launch<96, true, true>;
extern template struct Launch<128, false, true>;
extern template struct Launch<144, true, true>;
extern template struct Launch<192, true, true>;
extern template struct Launch<256, false, true>;
extern template struct Launch<288, true, false>;
extern template struct Launch<384, true, true>;
extern template struct Launch<512, false, true>;
extern template struct Launch<576, true, false>;
extern template struct Launch<768, true, true>;
extern template struct Launch<1152, true, false>;
extern template struct Launch<56, false, true>;
extern template struct Launch<60, false, true>;
extern template struct Launch<80, false, true>;
extern template struct Launch<84, true, true>;
extern template struct Launch<90, true, false>;
extern template struct Launch<100, false, true>;
extern template struct Launch<108, true, true>;
extern template struct Launch<112, false, true>;
extern template struct Launch<120, true, true>;
extern template struct Launch<126, true, false>;
extern template struct Launch<140, false, true>;
extern template struct Launch<150, true, false>;
extern template struct Launch<160, false, true>;
extern template struct Launch<162, true, false>;
extern template struct Launch<168, true, true>;
extern template struct Launch<180, true, true>;
extern template struct Launch<196, false, true>;
extern template struct Launch<200, false, true>;
extern template struct Launch<210, true, false>;
extern template struct Launch<216, true, true>;
extern template struct Launch<224, false, true>;
extern template struct Launch<240, true, true>;
extern template struct Launch<252, true, true>;
extern template struct Launch<270, true, false>;
extern template struct Launch<294, true, false>;
extern template struct Launch<300, true, false>;
extern template struct Launch<324, true, false>;
extern template struct Launch<336, true, false>;
extern template struct Launch<360, true, false>;
extern template struct Launch<378, true, false>;
template <int L, bool PADDED, bool GRID> static LenEntry entry() {
  return {L, PADDED, GRID, Launch<L, PADDED, GRID>::run, Len<L>::steps, {Len<L>::R(0), Len<L>::R(1), Len<L>::R(2)}};
}
static const LenEntry kLens[] = {entry<16, false, true>(),
                                 entry<24, true, true>(),
                                 entry<32, false, true>(),
                                 entry<48, true, true>(),
                                 entry<64, false, true>(),
                                 entry<72, true, true>(),
                                 entry<96, true, true>(),
                                 entry<128, false, true>(),
                                 entry<144, true, true>(),
                                 entry<192, true, true>(),
                                 entry<256, false, true>(),
                                 entry<288, true, false>(),
                                 entry<384, true, true>(),
                                 entry<512, false, true>(),
                                 entry<576, true, false>(),
                                 entry<768, true, true>(),
                                 entry<1152, true, false>(),
                                 entry<56, false, true>(),
                                 entry<60, false, true>(),
                                 entry<80, false, true>(),
                                 entry<84, true, true>(),
                                 entry<90, true, false>(),
                                 entry<100, false, true>(),
                                 entry<108, true, true>(),
                                 entry<112, false, true>(),
                                 entry<120, true, true>(),
                                 entry<126, true, false>(),
                                 entry<140, false, true>(),
                                 entry<150, true, false>(),
                                 entry<160, false, true>(),
                                 entry<162, true, false>(),
                                 entry<168, true, true>(),
                                 entry<180, true, true>(),
                                 entry<196, false, true>(),
                                 entry<200, false, true>(),
                                 entry<210, true, false>(),
                                 entry<216, true, true>(),
                                 entry<224, false, true>(),
                                 entry<240, true, true>(),
                                 entry<252, true, true>(),
                                 entry<270, true, false>(),
                                 entry<294, true, false>(),
                                 entry<300, true, false>(),
                                 entry<324, true, false>(),
                                 entry<336, true, false>(),
                                 entry<360, true, false>(),
                                 entry<378, true, false>()};
static const LenEntry *find_len(int L) {
  for (const LenEntry &e : kLens)
    if (e.L == L) return &e;
  return nullptr;
}
// B of an instance; an inverse transform takes the radices backwards
static int len_bits(const LenEntry &l, FxKind kind, bool forward, bool inverse) {
  int rev[3];
  for (int q = 0; q < l.steps; ++q) rev[q] = l.R[l.steps - 1 - q];
  int b = 60;
  if (forward) b = std::min(b, fx_bits(l.R, l.steps, kind));
  if (inverse) b = std::min(b, fx_bits(rev, l.steps, kind));
  return b;
}

static __global__ void k_fx_tables(int n, double *mode, double *rinv, double *root, int len) {
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
      const LArgs a{static_cast<const longlong2 *>(s.tw), len_bits(*l, FX_STRIDED, !s.inverse, s.inverse || s.truncate), s};
      return l->fn(op, &a, dim3(unsigned(s.outer * ((s.kc + 7) / 8)), unsigned(s.groups)), st);
    }
  }
  SArgs a;
  if (!fx_plan(s.L, FX_STRIDED, &a.c.p)) return cudaErrorInvalidValue;
  a.c.tw = static_cast<const longlong2 *>(s.tw);
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
      const LRows a{static_cast<const longlong2 *>(r.tw), len_bits(*l, kind, kind == FX_R2C, kind == FX_C2R), r};
      return l->fn(op, &a, dim3(unsigned((r.rows + 15) / 16), unsigned(r.count)), st);
    }
  }
  RArgs a;
  if (!fx_plan(r.L, kind, &a.c.p)) return cudaErrorInvalidValue;
  a.c.tw = static_cast<const longlong2 *>(r.tw);
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
