// 64-bit fixed-point pencil transforms of the plain FP64 form: the arithmetic,
// the in-register DFTs and the transform plans (the kernels and their launches
// are in fx64.cu).
//
// GB300 runs FP64 at two fused multiply-adds per SM and clock (measured 1.9)
// against 64 - 128 integer operations, so an FP64 FFT is bound by the FP64
// pipe and not by HBM: cuFFT's D2Z / Z2D ran at 0.13 TB/s (256^3, padded 384).
// A pencil (one 1D transform) is therefore transformed in 64-bit integers with
// one exponent per pencil: every value is scaled by the same power of two so
// that the largest |re|, |im| lies just below 2^B, and B leaves room for the
// growth of the steps, so that nothing can overflow (FxPlan::B).  Additions are
// exact; a multiplication by a twiddle or an internal constant is rounded at
// the last bit of a 61-63 bit integer.  The error is absolute and below
// 2^-53 of the pencil's rms at the lengths used, where an FP64 FFT's is a few
// 2^-53: measured against 64-bit references it is no larger than cuFFT's
// (fields 1e-16 - 1e-15 of their norm).  Multiplications (three 32x32+64
// products each, 12.7 a clock and SM measured) cost more than additions here,
// which is what the radices and the rotations below are chosen for.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

namespace fx {

#define FX_HD __host__ __device__ __forceinline__

// ---------------------------------------------------------------------------
// constants: cos, sin and tan of rational turns in fixed point
// ---------------------------------------------------------------------------
// 2 pi num / den in Q62 for 0 <= num / den <= 1/8
FX_HD constexpr __int128 q62_angle(int num, int den) {
  const __int128 two_pi_q96 = (__int128(0x6487ed511ULL) << 64) | __int128(0x0b4611a62633145cULL);
  return (two_pi_q96 / den * num) >> 34;
}
// cosine and sine of an angle below pi / 4 by their Taylor series, Q62
FX_HD constexpr __int128 q62_cos(__int128 a) {
  const __int128 one = __int128(1) << 62, a2 = (a * a) >> 62;
  __int128 term = one, sum = one;
  for (int k = 1; k < 14; ++k) {
    term = -((term * a2) >> 62) / ((2 * k - 1) * (2 * k));
    sum += term;
  }
  return sum;
}
FX_HD constexpr __int128 q62_sin(__int128 a) {
  const __int128 a2 = (a * a) >> 62;
  __int128 term = a, sum = a;
  for (int k = 1; k < 14; ++k) {
    term = -((term * a2) >> 62) / ((2 * k) * (2 * k + 1));
    sum += term;
  }
  return sum;
}
struct CS {
  __int128 c, s;
};
// cos and sin of 2 pi num / den, Q62, any num >= 0
FX_HD constexpr CS q62_turn(long long num, long long den) {
  num %= den;
  int quarter = int(4 * num / den);
  long long n4 = 4 * num - quarter * den;  // the rest of the quarter: n4 / (4 den) turns in [0, 1/4)
  const long long d4 = 4 * den;
  const bool mirror = 8 * n4 > d4;  // above an eighth: cos and sin change places
  if (mirror) n4 = d4 / 4 - n4;
  const __int128 two_pi_q96 = (__int128(0x6487ed511ULL) << 64) | __int128(0x0b4611a62633145cULL);
  const __int128 a = (two_pi_q96 / d4 * n4) >> 34;
  __int128 c = q62_cos(a), s = q62_sin(a);
  if (mirror) {
    const __int128 t = c;
    c = s;
    s = t;
  }
  for (; quarter > 0; --quarter) {
    const __int128 t = c;
    c = -s;
    s = t;
  }
  return {c, s};
}
// sin(2 pi num/den) and tan(pi num/den) in Q63, |num/den| <= 1/8 (both below 1)
FX_HD constexpr long long q63_sin(int num, int den) {
  return num < 0 ? -q63_sin(-num, den) : (long long)(2 * q62_sin(q62_angle(num, den)));
}
FX_HD constexpr long long q63_tan_half(int num, int den) {
  if (num < 0) return -q63_tan_half(-num, den);
  const __int128 c = q62_cos(q62_angle(num, 2 * den)), s = q62_sin(q62_angle(num, 2 * den));
  return (long long)((s << 63) / c);
}

// ---------------------------------------------------------------------------
// arithmetic
// ---------------------------------------------------------------------------
struct I2 {
  long long x, y;
};
FX_HD I2 operator+(I2 a, I2 b) { return {a.x + b.x, a.y + b.y}; }
FX_HD I2 operator-(I2 a, I2 b) { return {a.x - b.x, a.y - b.y}; }

// a W / 2^64, W = wh 2^32 + wl with wl signed: three signed 32-bit products;
// the fourth, a_lo wl 2^-64 (below a quarter in size, of either sign), is left out
FX_HD long long mulq(long long a, int wh, int wl) {
  const int al = int(a);
  const int ah = int(a >> 32) + int(unsigned(al) >> 31);  // a = ah 2^32 + al
  long long mid = (long long)ah * wl + (1LL << 31);
  mid += (long long)al * wh;
  return (long long)ah * wh + (mid >> 32);
}
FX_HD long long mulq(long long a, long long w) {
  const int wl = int(w);
  return mulq(a, int(w >> 32) + int(unsigned(wl) >> 31), wl);
}
// a w for a constant |w| < 1, W = w 2^63
template <long long W> FX_HD long long mulk(long long a) {
  constexpr int wl = int(W);
  constexpr int wh = int(W >> 32) + int(unsigned(wl) >> 31);
  return mulq(a + a, wh, wl);
}
template <long long W> FX_HD I2 mulk(I2 a) { return {mulk<W>(a.x), mulk<W>(a.y)}; }
FX_HD I2 minus_half(I2 a, I2 b) { return {a.x - (b.x >> 1), a.y - (b.y >> 1)}; }
FX_HD I2 minus_quarter(I2 a, I2 b) { return {a.x - (b.x >> 2), a.y - (b.y >> 2)}; }

// the same DFTs in single precision (fs32.cuh)
struct F2 {
  float x, y;
};
FX_HD F2 operator+(F2 a, F2 b) { return {a.x + b.x, a.y + b.y}; }
FX_HD F2 operator-(F2 a, F2 b) { return {a.x - b.x, a.y - b.y}; }
template <long long W> FX_HD F2 mulk(F2 a) {
  constexpr float w = float(double(W) * 1.0842021724855044e-19);  // 2^-63
  return {a.x * w, a.y * w};
}
FX_HD F2 minus_half(F2 a, F2 b) { return {a.x - 0.5f * b.x, a.y - 0.5f * b.y}; }
FX_HD F2 minus_quarter(F2 a, F2 b) { return {a.x - 0.25f * b.x, a.y - 0.25f * b.y}; }

// v exp(-2 pi i NUM / DEN): quarter turns by exchange, an eighth by one
// constant, the rest by three lifting steps (tan, sin, tan of an angle of at
// most pi/4: all constants below one, three products instead of four)
template <int NUM, int DEN> FX_HD I2 rotc(I2 v) {
  constexpr int n4 = 4 * (((NUM % DEN) + DEN) % DEN);
  constexpr int quarter = (n4 + DEN / 2) / DEN;
  constexpr int r = n4 - quarter * DEN;  // the rest: r / (4 DEN) turns, at most an eighth of one
  I2 q = v;
  if constexpr (quarter % 4 == 1) q = {v.y, -v.x};
  if constexpr (quarter % 4 == 2) q = {-v.x, -v.y};
  if constexpr (quarter % 4 == 3) q = {-v.y, v.x};
  constexpr long long h = 6521908912666391106LL;  // sqrt(1/2) 2^63
  if constexpr (r == 0) {
    return q;
  } else if constexpr (2 * r == DEN) {
    return {mulk<h>(q.x + q.y), mulk<h>(q.y - q.x)};
  } else if constexpr (2 * r == -DEN) {
    return {mulk<h>(q.x - q.y), mulk<h>(q.x + q.y)};
  } else {
    constexpr long long t = q63_tan_half(r, 4 * DEN), s = q63_sin(r, 4 * DEN);
    const long long x = q.x + mulk<t>(q.y);
    const long long y = q.y - mulk<s>(x);
    return {x + mulk<t>(y), y};
  }
}

template <int NUM, int DEN> FX_HD F2 rotc(F2 v) {
  constexpr int n = ((NUM % DEN) + DEN) % DEN;
  if constexpr (n == 0) return v;
  else if constexpr (4 * n == DEN) return {v.y, -v.x};
  else if constexpr (2 * n == DEN) return {-v.x, -v.y};
  else if constexpr (4 * n == 3 * DEN) return {-v.y, v.x};
  else {
    constexpr CS w = q62_turn(n, DEN);
    constexpr float c = float(double((long long)w.c) * 2.168404344971009e-19),  // 2^-62
        s = float(double((long long)w.s) * 2.168404344971009e-19);
    return {v.x * c + v.y * s, v.y * c - v.x * s};
  }
}

template <int... I, class F> FX_HD void sfor_(F &&f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F> FX_HD void sfor(F &&f) { sfor_(static_cast<F &&>(f), std::make_integer_sequence<int, N>{}); }

constexpr int gcd_(int a, int b) { return b ? gcd_(b, a % b) : a; }
constexpr int inv_mod(int a, int m) {
  for (int x = 1; x < m; ++x)
    if (a * x % m == 1) return x;
  return 1;
}
// the first factor of a composite radix: coprime factors need no rotations
// between them (prime-factor mapping), powers split as evenly as possible
constexpr int radix_split(int R) {
  switch (R) {
    case 4: return 2;
    case 6: return 2;
    case 8: return 2;
    case 9: return 3;
    case 10: return 2;
    case 12: return 3;
    case 14: return 2;
    case 15: return 3;
    case 16: return 4;
    case 18: return 2;
    case 20: return 4;
    case 21: return 3;
    case 24: return 3;
    default: return 1;  // prime
  }
}

// X[k] = sum_n v[n] exp(-2 pi i n k / R), in place
template <int R> struct Dft {
  template <class V> static FX_HD void run(V *v) {
    constexpr int A = radix_split(R), B = R / A;
    V t[R];
    if constexpr (gcd_(A, B) == 1) {
      constexpr int ea = B * inv_mod(B % A, A), eb = A * inv_mod(A % B, B);  // CRT idempotents
      sfor<B>([&](auto b) {
        V c[A];
        sfor<A>([&](auto a) { c[a] = v[(B * decltype(a)::value + A * decltype(b)::value) % R]; });
        Dft<A>::run(c);
        sfor<A>([&](auto a) { t[decltype(a)::value * B + decltype(b)::value] = c[a]; });
      });
      sfor<A>([&](auto a) {
        Dft<B>::run(t + decltype(a)::value * B);
        sfor<B>([&](auto b) {
          v[(ea * decltype(a)::value + eb * decltype(b)::value) % R] = t[decltype(a)::value * B + decltype(b)::value];
        });
      });
    } else {
      sfor<B>([&](auto b) {
        V c[A];
        sfor<A>([&](auto a) { c[a] = v[B * decltype(a)::value + decltype(b)::value]; });
        Dft<A>::run(c);
        sfor<A>([&](auto a) {
          t[decltype(a)::value * B + decltype(b)::value] = rotc<decltype(a)::value * decltype(b)::value, R>(c[a]);
        });
      });
      sfor<A>([&](auto a) {
        Dft<B>::run(t + decltype(a)::value * B);
        sfor<B>([&](auto b) { v[decltype(a)::value + A * decltype(b)::value] = t[decltype(a)::value * B + decltype(b)::value]; });
      });
    }
  }
};
template <> struct Dft<1> {
  template <class V> static FX_HD void run(V *) {}
};
template <> struct Dft<2> {
  template <class V> static FX_HD void run(V *v) {
    const V a = v[0], b = v[1];
    v[0] = a + b;
    v[1] = a - b;
  }
};
template <> struct Dft<3> {
  template <class V> static FX_HD void run(V *v) {
    constexpr long long s = 7987674492471257551LL;  // sin(pi/3) 2^63
    const V t = v[1] + v[2], d = mulk<s>(v[1] - v[2]);
    const V m = minus_half(v[0], t);
    v[0] = v[0] + t;
    v[1] = {m.x + d.y, m.y - d.x};
    v[2] = {m.x - d.y, m.y + d.x};
  }
};
template <> struct Dft<5> {
  template <class V> static FX_HD void run(V *v) {
    constexpr long long c = 5156021714044493573LL;   // sqrt(5)/4 2^63
    constexpr long long s1 = 8771948077865237882LL;  // sin(2 pi/5) 2^63
    constexpr long long s2 = 5421362059670026167LL;  // sin(pi/5) 2^63
    const V t1 = v[1] + v[4], t2 = v[2] + v[3], d1 = v[1] - v[4], d2 = v[2] - v[3];
    const V t = t1 + t2, b = mulk<c>(t1 - t2);
    const V a = minus_quarter(v[0], t);
    const V m1 = a + b, m2 = a - b;
    const V e1 = mulk<s1>(d1) + mulk<s2>(d2), e2 = mulk<s2>(d1) - mulk<s1>(d2);
    v[0] = v[0] + t;
    v[1] = {m1.x + e1.y, m1.y - e1.x};
    v[4] = {m1.x - e1.y, m1.y + e1.x};
    v[2] = {m2.x + e2.y, m2.y - e2.x};
    v[3] = {m2.x - e2.y, m2.y + e2.x};
  }
};
template <> struct Dft<7> {
  template <class V> static FX_HD void run(V *v) {
    // cos and sin of 2 pi j / 7 in Q63, j = 1, 2, 3
    constexpr long long c1 = 5750678403727967667LL, c2 = -2052393359867478633LL, c3 = -8309971062287876938LL;
    constexpr long long s1 = 7211122632928341039LL, s2 = 8992122843167040398LL, s3 = 4001871146622878209LL;
    const V t1 = v[1] + v[6], t2 = v[2] + v[5], t3 = v[3] + v[4];
    const V d1 = v[1] - v[6], d2 = v[2] - v[5], d3 = v[3] - v[4];
    const V m1 = v[0] + mulk<c1>(t1) + mulk<c2>(t2) + mulk<c3>(t3);
    const V m2 = v[0] + mulk<c2>(t1) + mulk<c3>(t2) + mulk<c1>(t3);
    const V m3 = v[0] + mulk<c3>(t1) + mulk<c1>(t2) + mulk<c2>(t3);
    const V e1 = mulk<s1>(d1) + mulk<s2>(d2) + mulk<s3>(d3);
    const V e2 = mulk<s2>(d1) - mulk<s3>(d2) - mulk<s1>(d3);
    const V e3 = mulk<s3>(d1) - mulk<s1>(d2) + mulk<s2>(d3);
    v[0] = v[0] + t1 + t2 + t3;
    v[1] = {m1.x + e1.y, m1.y - e1.x};
    v[6] = {m1.x - e1.y, m1.y + e1.x};
    v[2] = {m2.x + e2.y, m2.y - e2.x};
    v[5] = {m2.x - e2.y, m2.y + e2.x};
    v[3] = {m3.x + e3.y, m3.y - e3.x};
    v[4] = {m3.x - e3.y, m3.y + e3.x};
  }
};

// v / 8, rounded (the element that a step's twiddles leave alone)
FX_HD I2 eighth(I2 v) { return {(v.x + 4) >> 3, (v.y + 4) >> 3}; }

// v 2^S -> double, rounded to nearest; S + 1086 is the biased exponent of bit 63
FX_HD double to_double(long long v, int S) {
  const long long sg = v >> 63;
  const unsigned long long a = (unsigned long long)((v ^ sg) - sg);
#ifdef __CUDA_ARCH__
  const int lz = __clzll((long long)a);
#else
  const int lz = a ? __builtin_clzll(a) : 64;
#endif
  const unsigned long long n = a << (lz & 63);
  const unsigned long long q = (n >> 11) + ((n >> 10) & 1);
  const int e = S + 1086 - lz;
  unsigned long long r = ((unsigned long long)(e - 1) << 52) + q;
  r = (a == 0 || e <= 0) ? 0 : (e >= 2047 ? 0x7ff0000000000000ULL : r);
  r |= (unsigned long long)sg & 0x8000000000000000ULL;
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)r);
#else
  double o;
  __builtin_memcpy(&o, &r, 8);
  return o;
#endif
}

// ---------------------------------------------------------------------------
// plans
// ---------------------------------------------------------------------------
constexpr int kMaxSteps = 6;

struct FxPlan {
  int L;                // length
  int steps;            // Stockham steps
  int R[kMaxSteps];     // radix of a step
  int NS[kMaxSteps];    // product of the radices before it
  unsigned magic[kMaxSteps];  // ceil(2^32 / NS): j / NS by a multiplication
  int P, lgP;           // pencils per CTA
  int T;                // threads per CTA
  int B;                // largest component of the input lies below 2^B
  int smem;             // bytes
};

enum FxKind { FX_STRIDED = 0, FX_C2R = 1, FX_R2C = 2 };

// B of a transform of the given radices: a step of radix R lets a modulus grow
// by R, the twiddles after it take three bits off; a c2r pencil holds two rows,
// an r2c pencil's spectra are separated by sums.  62.7 bits at most
int fx_bits(const int *R, int steps, FxKind kind);

// false where a length has a prime factor above 7 or fits no CTA
bool fx_plan(int L, FxKind kind, FxPlan *p);
inline bool fx_supported(int L) {
  FxPlan p;
  return L >= 8 && L % 2 == 0 && fx_plan(L, FX_STRIDED, &p) && fx_plan(L, FX_C2R, &p) && fx_plan(L, FX_R2C, &p);
}

}  // namespace fx
