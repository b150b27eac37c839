// Single-precision pruned transforms (fs32.cuh): lengths without an instance
// (run-time radices up to 16) and the launches.
#include "fs32.cuh"

#include <algorithm>
#include <mutex>
#include <vector>

namespace fx {

namespace {
struct Core32 {
  FxPlan p;  // steps, radices, T; P pencils of 8-byte values
  const float2 *tw;
};

constexpr int kSmem32 = 220 * 1024;

// the plan of a length: the fixed-point transforms' factorisation, with pencils
// and threads for 8-byte values
bool plan32(int L, FxPlan *p) {
  if (!fx_plan(L, FX_STRIDED, p)) return false;
  for (int P : {16, 8, 4, 2}) {
    int need = 32;
    for (int q = 0; q < p->steps; ++q) need = std::max(need, P * (L / p->R[q]));
    const int T = (need + 31) / 32 * 32;
    if (T > 768 || L * P * 8 > kSmem32) continue;
    p->P = P;
    p->lgP = P == 16 ? 4 : (P == 8 ? 3 : (P == 4 ? 2 : 1));
    p->T = T;
    p->smem = L * P * 8;
    return true;
  }
  return false;
}
}  // namespace

struct SArgs32 {
  FxPlan p;
  Strided s;
};
struct RArgs32 {
  FxPlan p;
  Rows r;
};

__device__ __forceinline__ int slot32(int e, int q, int lgP) { return (e << lgP) + (q ^ (e & ((1 << lgP) - 1))); }

template <int R>
__device__ __noinline__ void step32(const float2 *tw, int L, int lgP, int NS, unsigned magic) {
  extern __shared__ __align__(16) F2 fsm[];
  const int t = threadIdx.x, nb = L / R, pen = t & ((1 << lgP) - 1), j = t >> lgP;
  const bool live = t < (nb << lgP);
  F2 v[R];
  int at = 0;
  if (live) {
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = fsm[slot32(j + r * nb, pen, lgP)];
    if (NS == 1) {
      at = j * R;
    } else {
      const int hi = int(__umulhi(unsigned(j), magic)), lo = j - hi * NS, inc = lo * (nb / NS);
      at = hi * NS * R + lo;
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], __ldg(&tw[r * inc]));
    }
    Dft<R>::run(v);
  }
  __syncthreads();
  if (live) {
#pragma unroll
    for (int r = 0; r < R; ++r) fsm[slot32(at + r * NS, pen, lgP)] = v[r];
  }
  __syncthreads();
}

__device__ __forceinline__ void transform32(const FxPlan &p, const float2 *tw) {
#pragma unroll 1
  for (int q = 0; q < p.steps; ++q) {
    const int L = p.L, lgP = p.lgP, NS = p.NS[q];
    const unsigned mg = p.magic[q];
    switch (p.R[q]) {
      case 2: step32<2>(tw, L, lgP, NS, mg); break;
      case 3: step32<3>(tw, L, lgP, NS, mg); break;
      case 4: step32<4>(tw, L, lgP, NS, mg); break;
      case 5: step32<5>(tw, L, lgP, NS, mg); break;
      case 6: step32<6>(tw, L, lgP, NS, mg); break;
      case 7: step32<7>(tw, L, lgP, NS, mg); break;
      case 8: step32<8>(tw, L, lgP, NS, mg); break;
      case 9: step32<9>(tw, L, lgP, NS, mg); break;
      case 10: step32<10>(tw, L, lgP, NS, mg); break;
      case 12: step32<12>(tw, L, lgP, NS, mg); break;
      case 14: step32<14>(tw, L, lgP, NS, mg); break;
      case 15: step32<15>(tw, L, lgP, NS, mg); break;
      case 16: step32<16>(tw, L, lgP, NS, mg); break;
    }
  }
}

__global__ void __launch_bounds__(768) k_fs_strided(const __grid_constant__ SArgs32 a) {
  mfx::pdl_begin();
  extern __shared__ __align__(16) F2 fsm[];
  const Strided &d = a.s;
  const float2 *tw = static_cast<const float2 *>(d.tw);
  const int L = a.p.L, lgP = a.p.lgP, P = 1 << lgP, T = blockDim.x, t = threadIdx.x;
  const int kblocks = (d.kc + P - 1) >> lgP;
  const int o = blockIdx.x / kblocks, kz0 = (blockIdx.x - o * kblocks) << lgP;
  const int pen = t & (P - 1), kz = kz0 + pen;
  const bool lv = kz < d.kc;
  const int n = d.n, nh = n >> 1, dl = T >> lgP;
  for (int op = d.first[blockIdx.y]; op < d.first[blockIdx.y + 1]; ++op) {
    const float2 *src = static_cast<const float2 *>(d.src[op]) + (long long)o * d.in_outer + kz;
    const int pr = d.pr[op];
    const bool scaled = (pr | d.pk[op]) != 0 || d.in_fac != 0.0;
    const float kf = scaled ? kz_factor(kz, n, d.pk[op], d.in_fac) : 1.f;
#pragma unroll 4
    for (int l = t >> lgP; l < L; l += dl) {
      F2 v = {0.f, 0.f};
      const int i = !d.pad_in ? l : (l <= nh ? l : (l > n ? l - nh : -1));
      if (lv && i >= 0) {
        v = ld(src + (long long)i * d.in_row);
        if (scaled) {
          const float f = row_factor(i, n, pr) * kf;
          v = {v.x * f, v.y * f};
        }
      }
      fsm[slot32(l, pen, lgP)] = swap_if(v, d.inverse);
    }
    __syncthreads();
    transform32(a.p, tw);
    bool inverse = d.inverse;
    if (d.truncate) {
      const float fac = float(d.fac);
      for (int l = t >> lgP; l < L; l += dl) {
        F2 &w = fsm[slot32(l, pen, lgP)];
        const F2 v = w;
        w = l < nh || l > n ? F2{v.y * fac, v.x * fac} : F2{0.f, 0.f};
      }
      __syncthreads();
      transform32(a.p, tw);
      inverse = true;
    }
    float2 *dst = static_cast<float2 *>(d.dst[op]) + (long long)o * d.out_outer + kz;
    const int so = o > nh ? o - n : o;
    for (int l = t >> lgP; l < L; l += dl) {
      const int i = !d.cut_out ? l : (l <= nh ? l : (l > n ? l - nh : -1));
      if (i < 0 || !lv) continue;
      F2 v = swap_if(fsm[slot32(l, pen, lgP)], inverse);
      if (d.cut_out) {
        if (i == nh || (d.inv_lap && o == nh)) {
          v = {0.f, 0.f};
        } else if (d.inv_lap) {
          const float f = lap_factor(d, so, i > nh ? i - n : i, kz);
          v = {v.x * f, v.y * f};
        }
      }
      dst[(long long)i * d.out_row] = make_float2(v.x, v.y);
    }
    if (d.inv_lap && kz0 + P >= d.kc) {
      float2 *z = static_cast<float2 *>(d.dst[op]) + (long long)o * d.out_outer + d.kc;  // the kz Nyquist column
      for (int i = t; i < n; i += T) z[(long long)i * d.out_row] = make_float2(0.f, 0.f);
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(768) k_fs_c2r_g(const __grid_constant__ RArgs32 a) {
  mfx::pdl_begin();
  extern __shared__ __align__(16) F2 fsm[];
  const Rows &d = a.r;
  const int L = a.p.L, lgP = a.p.lgP, P = 1 << lgP, T = blockDim.x, t = threadIdx.x, lane = t & 31;
  float *base = static_cast<float *>(d.field[blockIdx.y]);
  const long long row0 = (long long)blockIdx.x * 2 * P;
  const int h = L >> 1;
  for (int p = t >> 5; p < P; p += T >> 5) {
    const long long row = row0 + 2 * p;
    const bool la = row < d.rows, lb = row + 1 < d.rows;
    const float2 *sa = reinterpret_cast<const float2 *>(base + row * d.pitch);
    const float2 *sb = reinterpret_cast<const float2 *>(base + (row + 1) * d.pitch);
#pragma unroll 4
    for (int k = lane; k <= h; k += 32) {
      F2 x = {0.f, 0.f}, y = {0.f, 0.f};
      if (la && k < d.kc) x = ld(sa + k);
      if (lb && k < d.kc) y = ld(sb + k);
      // exchanged for the inverse transform; only the real parts at k = 0, L/2
      if (k == 0 || k == h) {
        fsm[slot32(k, p, lgP)] = {y.x, x.x};
      } else {
        fsm[slot32(k, p, lgP)] = {x.y + y.x, x.x - y.y};
        fsm[slot32(L - k, p, lgP)] = {y.x - x.y, x.x + y.y};
      }
    }
  }
  __syncthreads();
  transform32(a.p, static_cast<const float2 *>(d.tw));
  for (int p = t >> 5; p < P; p += T >> 5) {
    const long long row = row0 + 2 * p;
    float *da = base + row * d.pitch, *db = da + d.pitch;
    for (int e = lane; e < L; e += 32) {
      const F2 v = fsm[slot32(e, p, lgP)];
      if (row < d.rows) da[e] = v.y;
      if (row + 1 < d.rows) db[e] = v.x;
    }
  }
}

__global__ void __launch_bounds__(768) k_fs_r2c_g(const __grid_constant__ RArgs32 a) {
  mfx::pdl_begin();
  extern __shared__ __align__(16) F2 fsm[];
  const Rows &d = a.r;
  const int L = a.p.L, lgP = a.p.lgP, P = 1 << lgP, T = blockDim.x, t = threadIdx.x, lane = t & 31;
  float *base = static_cast<float *>(d.field[blockIdx.y]);
  const long long row0 = (long long)blockIdx.x * 2 * P;
  for (int p = t >> 5; p < P; p += T >> 5) {
    const long long row = row0 + 2 * p;
    const float *sa = base + row * d.pitch, *sb = sa + d.pitch;
#pragma unroll 4
    for (int e = lane; e < L; e += 32)
      fsm[slot32(e, p, lgP)] = {row < d.rows ? sa[e] : 0.f, row + 1 < d.rows ? sb[e] : 0.f};
  }
  __syncthreads();
  transform32(a.p, static_cast<const float2 *>(d.tw));
  for (int p = t >> 5; p < P; p += T >> 5) {
    const long long row = row0 + 2 * p;
    float2 *da = reinterpret_cast<float2 *>(base + row * d.pitch), *db = reinterpret_cast<float2 *>(base + (row + 1) * d.pitch);
    for (int k = lane; k < d.kc; k += 32) {
      const F2 u = fsm[slot32(k, p, lgP)], w = fsm[slot32(k ? L - k : 0, p, lgP)];
      if (row < d.rows) da[k] = make_float2(0.5f * (u.x + w.x), 0.5f * (u.y - w.y));
      if (row + 1 < d.rows) db[k] = make_float2(0.5f * (u.y + w.y), 0.5f * (w.x - u.x));
    }
  }
}

// ---------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------
using Len32Fn = cudaError_t (*)(FsOp, const Strided *, const Rows *, dim3, cudaStream_t);
struct Len32Entry {
  int L;
  bool padded, grid;
  Len32Fn fn;
};
#define FS_LENGTHS(X)                                                                                              \
  X(16, false, true) X(24, true, true) X(32, false, true) X(48, true, true) X(64, false, true) X(96, true, true)    \
  X(128, false, true) X(192, true, true) X(256, false, true) X(384, true, true) X(512, false, true) X(768, true, true) \
  X(56, false, true) \
  X(60, false, true) \
  X(72, true, true) \
  X(80, false, true) \
  X(84, true, true) \
  X(90, true, false) \
  X(100, false, true) \
  X(108, true, true) \
  X(112, false, true) \
  X(120, true, true) \
  X(126, true, false) \
  X(140, false, true) \
  X(144, true, true) \
  X(150, true, false) \
  X(160, false, true) \
  X(162, true, false) \
  X(168, true, true) \
  X(180, true, true) \
  X(196, false, true) \
  X(200, false, true) \
  X(210, true, false) \
  X(216, true, true) \
  X(224, false, true) \
  X(240, true, true) \
  X(252, true, true) \
  X(270, true, false) \
  X(294, true, false) \
  X(300, true, false) \
  X(324, true, false) \
  X(336, true, false) \
  X(360, true, false) \
  X(378, true, false)
#define FS_EXTERN(L, P, G) extern template struct Launch32<L, P, G>;
FS_LENGTHS(FS_EXTERN)
#define FS_ENTRY(L, P, G) {L, P, G, Launch32<L, P, G>::run},
static const Len32Entry kLens32[] = {FS_LENGTHS(FS_ENTRY)};
static const Len32Entry *find32(int L) {
  for (const Len32Entry &e : kLens32)
    if (e.L == L) return &e;
  return nullptr;
}

bool length_fast32(int L, bool padded) {
  const Len32Entry *e = find32(L);
  return (e && (padded ? e->padded : e->grid)) || (L <= 96 && length_supported(L));
}

cudaError_t prepare_device32(int dev) {
  static std::mutex mu;
  static std::vector<bool> done;
  std::lock_guard<std::mutex> lk(mu);
  if (dev < int(done.size()) && done[dev]) return cudaSuccess;
  for (const void *f : {(const void *)k_fs_strided, (const void *)k_fs_c2r_g, (const void *)k_fs_r2c_g}) {
    const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem32);
    if (e != cudaSuccess) return e;
  }
  for (const Len32Entry &l : kLens32) {
    const cudaError_t e = l.fn(FS_PREPARE, nullptr, nullptr, dim3(), nullptr);
    if (e != cudaSuccess) return e;
  }
  if (dev >= int(done.size())) done.resize(dev + 1, false);
  done[dev] = true;
  return cudaSuccess;
}

cudaError_t run_strided32(const Strided &s, cudaStream_t st) {
  if (const Len32Entry *l = find32(s.L)) {
    const bool p = l->padded && 3 * s.n == 2 * s.L;
    FsOp op = FS_PREPARE;
    if (s.inverse && !s.cut_out && !s.truncate)
      op = s.pad_in ? (p ? FS_INV_PAD : op) : (l->grid && s.in_fac == 0.0 ? FS_INV : op);
    else if (!s.inverse && !s.pad_in && s.groups == s.ops && p)
      op = s.truncate ? FS_TRUNC : (s.cut_out ? FS_CUT : op);
    if (op != FS_PREPARE)
      return l->fn(op, &s, nullptr, dim3(unsigned(s.outer * ((s.kc + 15) / 16)), unsigned(s.groups)), st);
  }
  SArgs32 a;
  if (!plan32(s.L, &a.p)) return cudaErrorInvalidValue;
  a.s = s;
  const int kb = (s.kc + a.p.P - 1) / a.p.P;
  mfx::launch_pdl(k_fs_strided, dim3(unsigned(s.outer * kb), unsigned(s.groups)), a.p.T, a.p.smem, st, a);
  return cudaGetLastError();
}

static cudaError_t rows32(const Rows &r, bool inverse, cudaStream_t st) {
  if (const Len32Entry *l = find32(r.L)) {
    FsOp op = FS_PREPARE;
    if (inverse) op = l->padded && r.kc <= r.L / 3 + 1 ? FS_C2R_PAD : (l->grid ? FS_C2R : op);
    else if (l->padded && r.kc <= r.L / 3) op = FS_R2C;
    if (op != FS_PREPARE) return l->fn(op, nullptr, &r, dim3(unsigned((r.rows + 31) / 32), unsigned(r.count)), st);
  }
  RArgs32 a;
  if (!plan32(r.L, &a.p)) return cudaErrorInvalidValue;
  a.r = r;
  const long long per = 2 * a.p.P;
  const dim3 grid(unsigned((r.rows + per - 1) / per), unsigned(r.count));
  if (inverse) mfx::launch_pdl(k_fs_c2r_g, grid, a.p.T, a.p.smem, st, a);
  else mfx::launch_pdl(k_fs_r2c_g, grid, a.p.T, a.p.smem, st, a);
  return cudaGetLastError();
}
cudaError_t run_c2r32(const Rows &r, cudaStream_t st) { return rows32(r, true, st); }
cudaError_t run_r2c32(const Rows &r, cudaStream_t st) { return rows32(r, false, st); }

}  // namespace fx
