// Fixed-point transforms of the lengths 16, 24, 32, 48, 64, 72, 96 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template struct Launch<16, false, true>;
template struct Launch<24, true, true>;
template struct Launch<32, false, true>;
template struct Launch<48, true, true>;
template struct Launch<64, false, true>;
template struct Launch<72, true, true>;
template struct Launch<96, true, true>;
}  // namespace fx
