// Box-Muller in 64-bit fixed point for the plain FP64 form's white noise.
//
// z = sqrt(-ln u_b) exp(2 pi i u_a) of two 48-bit variates (random_ngenic.cc:
// 117-121).  CUDA's double-precision log, sincos and sqrt keep the FP64 pipe
// (1.9 operations per SM and clock) busy for about 100 operations a mode; the
// tables and short series below take 19 products of three 32-bit
// multiplications each and leave one square root to it.
//  * cos, sin: 512 directions from a table, the remaining angle (at most
//    2 pi / 1024) by its Taylor series to the sixth order (the next term is below
//    2^-64), and one rotation.
//  * -ln u: u = m 2^e, m in [1, 2), times the reciprocal of the middle c of m's
//    1/256th of the interval gives 1 + r, |r| < 2^-9; ln m = ln c + log1p(r), its
//    series to r^6 (the next term is below 2^-65).
// Errors are a few 2^-62 in cos, sin and -ln u.  Where -ln u lies below 2^-10
// (u within 1e-3 of one) that would show in the square root's 53 bits: those
// modes take log().  Against 64-bit-mantissa arithmetic the noise of 64^3 is off
// by 8e-17 of its norm (with CUDA's double functions 2.4e-16).  256^3: 1.45 ->
// 0.36 ms with the generator's blocks, 64^3 118 -> 31 us.
#pragma once
#include "fx64.cuh"
#include "ranlxd.cuh"

namespace mfx {

struct NoiseTables {
  long long cs[512][2];  // cos, sin of 2 pi h / 512, Q62
  long long lc[256][2];  // 1 / c in Q63, ln c in Q62, c = 1 + (i + 1/2) / 256
};
constexpr long long noise_ln(int num, int den) {
  // ln(num / den) = 2 artanh((num - den) / (num + den)), Q62
  const __int128 y = (__int128(num - den) << 62) / (num + den), y2 = (y * y) >> 62;
  __int128 term = y, sum = 0;
  for (int k = 1; k < 60; k += 2) {
    sum += term / k;
    term = (term * y2) >> 62;
  }
  return (long long)(2 * sum);
}
constexpr NoiseTables make_noise_tables() {
  NoiseTables t{};
  for (int h = 0; h < 512; ++h) {
    const fx::CS w = fx::q62_turn(h, 512);
    t.cs[h][0] = (long long)w.c;
    t.cs[h][1] = (long long)w.s;
  }
  for (int i = 0; i < 256; ++i) {
    t.lc[i][0] = (long long)(((__int128(1) << 63) * 512) / (513 + 2 * i));
    t.lc[i][1] = noise_ln(513 + 2 * i, 512);
  }
  return t;
}
static __device__ constexpr NoiseTables kNoise = make_noise_tables();

// cos and sin of 2 pi a / 2^48, Q62
__device__ __forceinline__ void noise_direction(uint64_t a, long long &c, long long &s) {
  using fx::mulq;
  constexpr long long kPi4 = 7244019458077122842LL;            // pi / 4 in Q63
  constexpr long long k120 = 153722867280912930LL;             // 2^64 / 120
  constexpr long long k720 = 25620477880152155LL;              // 2^64 / 720
  constexpr long long k6 = 768614336404564651LL, k24 = 192153584101141163LL;  // 1/6, 1/24 in Q62
  const uint64_t h = (a + (uint64_t(1) << 38)) >> 39;
  const long long rem = (long long)a - (long long)(h << 39);
  const long long th = mulq(rem << 24, kPi4);                  // the rest of the angle, Q68
  const long long p = mulq(th, th), p62 = p >> 10;             // its square, Q72 and Q62
  const long long t3 = mulq(th, mulq(p62, k6 - mulq(p62, k120)));            // th - sin, Q64
  const long long sn = th - (t3 << 4);                                       // sin, Q68
  const long long cm = -mulq(p, (1LL << 59) - mulq(p62, k24 - mulq(p62, k720)));  // cos - 1, Q68
  const longlong2 w = __ldg(reinterpret_cast<const longlong2 *>(kNoise.cs[h & 511]));
  c = w.x + ((mulq(w.x, cm) - mulq(w.y, sn) + 8) >> 4);
  s = w.y + ((mulq(w.y, cm) + mulq(w.x, sn) + 8) >> 4);
}

// sqrt(-ln(b 2^-48)), 0 < b < 2^48
__device__ __forceinline__ double noise_amplitude(uint64_t b) {
  using fx::mulq;
  constexpr long long kLn2 = 3196577161300663915LL;  // ln 2 in Q62
  constexpr long long kLn2Q57 = 99893036290645747LL;
  constexpr long long c2 = 1LL << 59;                // the series' coefficients in Q60
  constexpr long long c3 = -384307168202282325LL, c4 = 288230376151711744LL, c5 = -230584300921369395LL,
                      c6 = 192153584101141163LL;
  const int lz = __clzll((long long)b);              // at least 16
  const uint64_t m = b << lz;                        // mantissa in [1, 2), Q63
  const longlong2 t = __ldg(reinterpret_cast<const longlong2 *>(kNoise.lc[(m >> 55) & 255]));
  const long long r = mulq((long long)(m >> 1), t.x) - (1LL << 61);  // Q61, |r| < 2^-9
  const long long rq = r << 9, r64 = r << 3;
  const long long r2 = mulq(rq, rq);                 // Q76
  long long q = c5 + mulq(r64, c6);
  q = c4 + mulq(r64, q);
  q = c3 + mulq(r64, q);
  q = c2 + mulq(r64, q);
  const long long lnm = t.y + (r << 1) - ((mulq(r2, q) + 512) >> 10);  // ln m, Q62
  // -ln u = (lz - 15) ln 2 - ln m: Q62 below ln 2, else Q57
  const bool near = lz == 16;
  const long long x = near ? kLn2 - lnm : (long long)(lz - 15) * kLn2Q57 - ((lnm + 16) >> 5);
  if (near && x < (1LL << 52)) return sqrt(-log(double(b) * kTwoM48));
  return sqrt(fx::to_double(x, near ? -62 : -57));
}

}  // namespace mfx
