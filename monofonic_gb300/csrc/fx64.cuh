// 64-bit fixed-point pencil transforms of the plain FP64 form: the arithmetic,
// the in-register DFTs, the scale of a pencil and the transform plans (the
// kernels and their launches are in fx64.cu and fx64_len.cuh).
//
// GB300 runs FP64 at two fused multiply-adds per SM and clock (measured 1.9)
// against 64 - 128 integer operations, so an FP64 FFT is bound by the FP64
// pipe and not by HBM: cuFFT's D2Z / Z2D ran at 0.13 TB/s (256^3, padded 384).
// A pencil (one 1D transform) is therefore transformed in 64-bit integers with
// one exponent per pencil: every value is scaled by the same power of two,
// chosen from the pencil's sum of magnitudes and its largest component so that
// no intermediate can leave 64 bits (pencil_scale).  Additions are
// exact; a multiplication by a twiddle or an internal constant is rounded at
// the last bit of a 61-63 bit integer.  What is lost is absolute, a few units
// of the last place for every step.  Against long double, relative to the
// output's norm and rounded to double, pencils with amplitudes from flat to k^-4
// are off by 5e-17 to 1.0e-16 in two steps, to 1.5e-16 in three and as c2r to
// 1.8e-16; numpy's FP64 transforms of them by 1.1e-16 to 2.8e-16, and in no case
// by less (tests/test_fx64_range.py).  Multiplications (three 32x32+64
// products each, 12.7 a clock and SM measured) cost more than additions here,
// which is what the radices and the rotations below are chosen for.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
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
// Halves and quarters are rounded to even: an offset, as of a floor, would be the
// same in every pencil, and the passes that follow would sum it over the grid into
// the modes along an axis (phi(2)'s lowest modes at 288^3 were off by 4e-15 of its
// norm, with cuFFT by 5e-16).
FX_HD long long minus_half(long long a, long long b) {
  const long long h = b >> 1;
  return a - h - (h & b & 1);
}
FX_HD long long minus_quarter(long long a, long long b) {
  const long long h = b >> 2;
  return a - h - ((b >> 1) & (b | h) & 1);
}
FX_HD I2 minus_half(I2 a, I2 b) { return {minus_half(a.x, b.x), minus_half(a.y, b.y)}; }
FX_HD I2 minus_quarter(I2 a, I2 b) { return {minus_quarter(a.x, b.x), minus_quarter(a.y, b.y)}; }

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

// Twiddle constants are held as w 2^62, so a product with one is a quarter of
// v w; the element that a step's twiddles leave alone is quartered like them.
// Three products: c = cos, s = -sin, the constants c, s + c and s - c split into
// signed halves (hi, lo)
FX_HD long long quarter(long long v) { return (v + 1 + ((v >> 2) & 1)) >> 2; }
FX_HD I2 quarter(I2 v) { return {quarter(v.x), quarter(v.y)}; }
// v 2^k, rounded, halves away from zero: modes of either sign, no offset
FX_HD long long rescale(long long v, int k) {
  const int dn = k < 0 ? -k : 0;
  const long long half = dn ? (1LL << (dn - 1)) + (v >> 63) : 0;
  return dn ? (v + half) >> dn : v << k;
}
FX_HD I2 twiddle4(I2 v, int4 c_p, int2 m) {
  const long long k = mulq(v.x + v.y, c_p.x, c_p.y);
  return {k - mulq(v.y, c_p.z, c_p.w), k + mulq(v.x, m.x, m.y)};
}
// The constants of (cos, -sin)(2 pi t / L).  Powers of two (1, 1/2) are one unit
// smaller: their products would end in halves, which mulq rounds up, an offset in
// the modes 0 of all pencils; so these halves round towards zero.
inline void twiddle_constants(int t, int L, int4 *c_p, int2 *m) {
  const CS w = q62_turn(t, L);
  auto inexact = [](long long v) { return (v & 0xffffffffLL) || v == 0 ? v : (v > 0 ? v - 1 : v + 1); };
  const long long c = inexact((long long)w.c), s = inexact((long long)-w.s);
  auto lo = [](long long w) { return int(w); };
  auto hi = [](long long w) { return int(w >> 32) + int(unsigned(int(w)) >> 31); };
  *c_p = make_int4(hi(c), lo(c), hi(s + c), lo(s + c));
  *m = make_int2(hi(s - c), lo(s - c));
}

// ---------------------------------------------------------------------------
// scale of a pencil
// ---------------------------------------------------------------------------
// log2 v in Q20, rounded up
FX_HD constexpr int log2_q20(int v) {
  double m = v;
  int r = 0;
  for (; m >= 2.0; m *= 0.5) r += 1 << 20;
  for (int bit = 1 << 19; bit; bit >>= 1)
    if ((m *= m) >= 2.0) {
      m *= 0.5;
      r += bit;
    }
  return r + 1;
}
// The power k of two that a pencil's values are multiplied by.  `top` is the high
// word of its largest component, `sum` a high word without the bias of its sum of
// magnitudes (or of a bound of it); a double's high word, taken as a number, is a
// logarithm to base 2 in Q20 that is low by at most 0.0861.  Every intermediate of step q is a sum of inputs times
// factors of modulus at most one, each input once, over 2^bits_lost(q): its
// modulus stays below the pencil's sum of magnitudes, and below the product of the
// radices so far times sqrt(2) times the largest component (lg[q], its logarithm).  The
// largest operand that the arithmetic makes of an intermediate of modulus A is
// 2 sqrt(2) A (the doubled sum of both components in an eighth turn), so
// A < 2^61.5 keeps all of them below 2^63.  The first bound is the smaller one
// where a few modes hold the pencil, the steep spectra of potentials and
// displacements, which then keep all their bits; the second one is for flat
// spectra, whose sums grow by the root of the length.  Scaled by the second bound
// alone, less what the steps lose, a flat pencil at length 72 left the range, and
// k^-2 pencils were off by 2e-16 at length 256 and 4e-16 at 384.  The sums cost 1%
// of a 256^3 3LPT pass (27.9 -> 28.2 ms) and 3% at 64^3 (203 -> 209 us).
// The twiddles of a step quarter its inputs.  Of three steps, where an intermediate
// of few large terms has not grown yet, the second one's are doubled before (half
// lost): k^-1 spectra of three-step c2r transforms are off by up to 1.8e-16 so,
// 2.7e-16 with quarters only, numpy's FP64 transforms of them by 2.3e-16.
FX_HD constexpr int bits_lost(int q, int steps) { return q == 0 ? 0 : (steps > 2 ? 2 * q - 1 : 2 * q); }
constexpr bool doubled(int q, int steps) { return q == 1 && steps > 2; }
constexpr int kScaleTop = int((61.5 - 0.0862) * 1048576.0);
template <class G> FX_HD int pencil_scale(int top, int sum, int steps, G lg) {
  const int m = top - 0x3ff00000 + 1, s = sum + 1;
  int v = -0x7fffffff;
#pragma unroll
  for (int q = 0; q < steps; ++q) {
    const int g = m + lg(q);
    const int b = (s < g ? s : g) - (bits_lost(q, steps) << 20);
    v = b > v ? b : v;
  }
  return (kScaleTop - v) >> 20;
}
// Magnitudes are summed in single precision, whose pipe is idle in these kernels
// (FP64 additions made the passes 14% longer at 256^3, a third at 64^3): high words
// relative to a base 120 binades below the largest one are moved to a float's
// place.  What lies below the base counts as it, which is nothing.
FX_HD int sum_base(int top) { return (top & 0x7ff00000) - (120 << 20); }
FX_HD float as_float(int b) {
#ifdef __CUDA_ARCH__
  return __int_as_float(b);
#else
  float f;
  __builtin_memcpy(&f, &b, 4);
  return f;
#endif
}
FX_HD int as_int(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_int(f);
#else
  int b;
  __builtin_memcpy(&b, &f, 4);
  return b;
#endif
}
FX_HD float sum_term(int word, int base) { return as_float(((word > base ? word : base) - base) << 3); }
// a sum taken to the base of `top`, brought to the base of a larger `to`
FX_HD float sum_rebase(float f, int top, int to) {
  const int e = 127 - ((to >> 20) - (top >> 20));
  return f * as_float(e > 0 ? e << 23 : 0);
}
// the high word without the bias of a sum
FX_HD int sum_word(float f, int top) { return (as_int(f) >> 3) + (sum_base(top) - 0x3ff00000); }
constexpr int kSqrt2 = 1 << 19, kTwice = 1 << 20;  // added to a sum's word: times sqrt(2), times two

// conversion of a pencil whose largest component has the biased exponent em:
// scale -> right shift of to_fixed_p.  A pencil whose values all lie below
// 2^-959 counts as zero.
FX_HD int shift_of(int em, int k) { return em < 64 ? 8192 : 1085 - k; }
FX_HD long long to_fixed_p(long long b, int sh) {
  const int d0 = sh - (int(b >> 52) & 0x7ff), d = d0 < 63 ? d0 : 63;
  const long long m = (long long)(((unsigned long long)((b & 0xfffffffffffffLL) | 0x10000000000000LL) << 10) >> d);
  const long long sg = b >> 63;
  return (m ^ sg) - sg;
}
// rounded: for c2r transforms of three steps, whose values are sums of two
FX_HD long long to_fixed_r(long long b, int sh) {
  const long long t = to_fixed_p(b & 0x7fffffffffffffffLL, sh - 1), m = (t + 1) >> 1, sg = b >> 63;
  return (m ^ sg) - sg;
}

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
  int lg[kMaxSteps];    // growth bound after a step (pencil_scale)
  int smem;             // bytes
};

// a c2r pencil's components are sums of two of its rows' components
enum FxKind { FX_STRIDED = 0, FX_C2R = 1, FX_R2C = 2 };

constexpr int kSmemMax = 220 * 1024;

// rough cost of a point: real multiplications (three products each, measured
// 4 a clock) and the shared-memory round trip of a step
inline double radix_cost(int R) {
  switch (R) {
    case 2: case 4: return 0.0;
    case 3: return 0.67; case 5: return 2.0; case 6: return 0.67; case 7: return 5.1;
    case 8: return 0.5; case 9: return 2.0; case 10: return 2.0; case 12: return 0.67;
    case 14: return 5.1; case 15: return 2.67; default: return 1.25;  // 16
  }
}

// best factorisation: fewest steps, then least cost, then smallest largest radix
inline void plan_search(int rest, int depth, double cost, int *cur, int &best_n, double &best_c, int *best) {
  constexpr int kRadices[] = {16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
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
      plan_search(rest / R, depth + 1, cost + radix_cost(R), cur, best_n, best_c, best);
    }
}

// lg of a step: the radices up to it, sqrt(2), and 2 for a c2r pencil
FX_HD constexpr int growth(int radices, FxKind kind) { return log2_q20(radices) + (1 << 19) + (kind == FX_C2R ? 1 << 20 : 0); }

// false where a length has a prime factor above 7 or fits no CTA
inline bool fx_plan(int L, FxKind kind, FxPlan *p) {
  *p = FxPlan{};
  p->L = L;
  int cur[kMaxSteps], best[kMaxSteps], n = kMaxSteps + 1;
  double c = 1e30;
  plan_search(L, 0, 0.0, cur, n, c, best);
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
    p->lg[q] = growth(ns, kind);
  }
  for (int P : {8, 4, 2, 1}) {
    int need = 32;  // threads: a butterfly each
    for (int q = 0; q < n; ++q) need = std::max(need, P * (L / p->R[q]));
    const int T = (need + 31) / 32 * 32;
    // pencils, then a number for each warp and pencil, or two for each row
    const int smem = L * P * 16 + std::max(T / 32, 4) * P * 4;
    if (T > 768 || smem > kSmemMax) continue;
    p->P = P;
    p->lgP = P == 8 ? 3 : (P == 4 ? 2 : P - 1);
    p->T = T;
    p->smem = smem;
    return true;
  }
  return false;
}
inline bool fx_supported(int L) {
  FxPlan p;
  return L >= 8 && L % 2 == 0 && fx_plan(L, FX_STRIDED, &p) && fx_plan(L, FX_C2R, &p) && fx_plan(L, FX_R2C, &p);
}

}  // namespace fx
