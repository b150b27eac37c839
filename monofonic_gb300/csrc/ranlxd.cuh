// RANLUX "ranlxd1" stream on 48-bit integer words, usable on host and device.
//
// monofonIC's NGenIC plugin draws its white noise from GSL's gsl_rng_ranlxd1
// (src/plugins/random_ngenic.cc:44-45, 104-114).  GSL is not part of the
// reference tree; the generator is restated here from M. Luescher's published
// RANLUX algorithm (Comput. Phys. Commun. 79 (1994) 100, double-precision
// variant, luxury level 1):
//   y[n] = y[n-5] - y[n-12] - c[n-1] mod 2^48, c[n] the borrow;
//   per block 202 words are generated and the last 12 delivered in order;
//   a delivered word y maps to the uniform y * 2^-48 (exact in a double);
//   the 12 seed words come from a 31-bit shift register holding the low 31
//   seed bits: each output bit is the complement of register bit b[i], after
//   which b[i] <- b[i] xor b[i+18 mod 31] and i advances (mod 31), 48 bits per
//   word, most significant first; seed 0 means seed 1.
//
// The device keeps the 12-word history as a sliding register window so that a
// fully unrolled block uses static register indices only.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define MFX_HD __host__ __device__ __forceinline__
#else
#define MFX_HD inline
#endif

namespace mfx {

static constexpr uint64_t kMask48 = (uint64_t(1) << 48) - 1;
static constexpr double kTwoM48 = 1.0 / 281474976710656.0;  // 2^-48

// the lower 48 bits in reverse order
MFX_HD uint64_t reverse48(uint64_t v) {
#ifdef __CUDA_ARCH__
  return __brevll(v) >> 16;
#else
  v = ((v >> 1) & 0x5555555555555555ULL) | ((v & 0x5555555555555555ULL) << 1);
  v = ((v >> 2) & 0x3333333333333333ULL) | ((v & 0x3333333333333333ULL) << 2);
  v = ((v >> 4) & 0x0f0f0f0f0f0f0f0fULL) | ((v & 0x0f0f0f0f0f0f0f0fULL) << 4);
  return __builtin_bswap64(v) >> 16;
#endif
}

struct Ranlxd1 {
  uint64_t w[12];  // y[n-12] .. y[n-1], oldest first
  uint64_t o[12];  // words of the current block still to be delivered, o[0] next
  uint32_t carry;
  int avail;

  // Seed from a value 0 <= v < 2^31 (all NGenIC column seeds are below
  // 0x7fffffff).  The 31-bit register is rotated so that bit 0 is always the
  // current tap b[i] and bit 18 the tap b[i+18].
  MFX_HD void seed31(uint32_t v) {
    if (v == 0) v = 1;
    uint32_t reg = v & 0x7fffffffu;
    // Twelve register bits at a time: the taps are 18 bits apart, so the first
    // 13 updates read no bit that another of them writes (bit by bit the seeding
    // was a chain of 576 dependent steps, a third of the noise kernel's time at
    // 32^3).  Fully unrolled over the 12 words so that w[] stays in registers.
#pragma unroll
    for (int q = 0; q < 12; ++q) {
      uint64_t word = 0;  // the 48 bits, the first one lowest
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        word |= uint64_t(~reg & 0xfffu) << (12 * l);
        reg = (reg >> 12) | (((reg ^ (reg >> 18)) & 0xfffu) << 19);
      }
      w[q] = reverse48(word);
    }
    carry = 0;
    avail = 0;
  }

  MFX_HD void block() {
#pragma unroll
    for (int t = 0; t < 202; ++t) {
      uint64_t d = w[7] - w[0] - uint64_t(carry);
      carry = uint32_t(d >> 63);
      d &= kMask48;
#pragma unroll
      for (int q = 0; q < 11; ++q) w[q] = w[q + 1];
      w[11] = d;
    }
#pragma unroll
    for (int q = 0; q < 12; ++q) o[q] = w[q];
    avail = 12;
  }

  MFX_HD uint64_t next() {
    if (avail == 0) block();
    const uint64_t v = o[0];
#pragma unroll
    for (int q = 0; q < 11; ++q) o[q] = o[q + 1];
    --avail;
    return v;
  }

  MFX_HD double uniform() { return double(next()) * kTwoM48; }
};

#if defined(__CUDACC__)
// The same stream a block (12 words) at a time, for kernels: the words are held
// in the upper 48 bits of register pairs, so that the borrow of a step is the
// hardware's borrow out of bit 63 and goes into the next step's subtraction as
// it is (three instructions a step, six with the borrow taken out of bit 48 by
// hand), and a round of twelve steps overwrites the twelve words in place.
struct RanlxdBlocks {
  uint32_t lo[12], hi[12];  // oldest first; the lower half of lo is zero
  uint32_t borrow;          // 0 or 0xffffffff

  __device__ __forceinline__ void seed31(uint32_t v) {
    Ranlxd1 r;
    r.seed31(v);
#pragma unroll
    for (int q = 0; q < 12; ++q) {
      lo[q] = uint32_t(r.w[q]) << 16;
      hi[q] = uint32_t(r.w[q] >> 16);
    }
    borrow = 0;
  }
  // word q of the last block
  __device__ __forceinline__ uint64_t word(int q) const { return (uint64_t(hi[q]) << 16) | (lo[q] >> 16); }

#define MFX_RLX_STEP(A, AH, B, BH)             \
  "subc.cc.u32 %" #A ", %" #B ", %" #A ";\n\t"  \
  "subc.cc.u32 %" #AH ", %" #BH ", %" #AH ";\n\t" \
  "and.b32 %" #A ", %" #A ", 0xffff0000;\n\t"
#define MFX_RLX_TEN                                                                                        \
  MFX_RLX_STEP(0, 12, 7, 19) MFX_RLX_STEP(1, 13, 8, 20) MFX_RLX_STEP(2, 14, 9, 21) MFX_RLX_STEP(3, 15, 10, 22) \
  MFX_RLX_STEP(4, 16, 11, 23) MFX_RLX_STEP(5, 17, 0, 12) MFX_RLX_STEP(6, 18, 1, 13) MFX_RLX_STEP(7, 19, 2, 14) \
  MFX_RLX_STEP(8, 20, 3, 15) MFX_RLX_STEP(9, 21, 4, 16)
#define MFX_RLX_OPS                                                                                          \
  "+r"(lo[0]), "+r"(lo[1]), "+r"(lo[2]), "+r"(lo[3]), "+r"(lo[4]), "+r"(lo[5]), "+r"(lo[6]), "+r"(lo[7]),        \
      "+r"(lo[8]), "+r"(lo[9]), "+r"(lo[10]), "+r"(lo[11]), "+r"(hi[0]), "+r"(hi[1]), "+r"(hi[2]), "+r"(hi[3]),  \
      "+r"(hi[4]), "+r"(hi[5]), "+r"(hi[6]), "+r"(hi[7]), "+r"(hi[8]), "+r"(hi[9]), "+r"(hi[10]), "+r"(hi[11]),  \
      "+r"(borrow)
  // 202 steps: sixteen rounds of twelve and ten more, after which the oldest
  // word is number ten; the words are put back in order
  __device__ __forceinline__ void block() {
#pragma unroll 4
    for (int round = 0; round < 16; ++round)
      asm("{\n\t.reg .u32 t;\n\tsub.cc.u32 t, 0, %24;\n\t" MFX_RLX_TEN MFX_RLX_STEP(10, 22, 5, 17)
              MFX_RLX_STEP(11, 23, 6, 18) "subc.u32 %24, 0, 0;\n\t}"
          : MFX_RLX_OPS);
    asm("{\n\t.reg .u32 t;\n\tsub.cc.u32 t, 0, %24;\n\t" MFX_RLX_TEN "subc.u32 %24, 0, 0;\n\t}" : MFX_RLX_OPS);
    const uint32_t l10 = lo[10], l11 = lo[11], h10 = hi[10], h11 = hi[11];
#pragma unroll
    for (int q = 11; q >= 2; --q) {
      lo[q] = lo[q - 2];
      hi[q] = hi[q - 2];
    }
    lo[0] = l10;
    lo[1] = l11;
    hi[0] = h10;
    hi[1] = h11;
  }
#undef MFX_RLX_STEP
#undef MFX_RLX_TEN
#undef MFX_RLX_OPS
};
#endif

// Host-side seeding for arbitrary `unsigned long` seeds, mirroring the 32-bit
// signed-integer arithmetic of the published seeding routine for seeds that do
// not fit in 31 bits.
inline void ranlxd1_seed_any(Ranlxd1 &r, unsigned long s) {
  if (s == 0) s = 1;
  int32_t v = int32_t(uint32_t(s & 0xffffffffUL));
  if (v >= 0) {
    r.seed31(uint32_t(v));
    return;
  }
  int bits[31];
  for (int q = 0; q < 31; ++q) { bits[q] = v % 2; v /= 2; }
  int ib = 0, jb = 18;
  for (int q = 0; q < 12; ++q) {
    // the published routine accumulates in a double; all partial values are
    // integers below 2^49 in magnitude, so int64 arithmetic is exact
    int64_t x = 0;
    for (int l = 0; l < 48; ++l) {
      x = 2 * x + int64_t((bits[ib] + 1) % 2);
      bits[ib] = (bits[ib] + bits[jb]) % 2;
      ib = (ib + 1) % 31;
      jb = (jb + 1) % 31;
    }
    r.w[q] = uint64_t(x) & kMask48;
  }
  r.carry = 0;
  r.avail = 0;
}

}  // namespace mfx
