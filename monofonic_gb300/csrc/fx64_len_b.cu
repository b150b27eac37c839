// Fixed-point transforms of the lengths 128, 144, 192, 256 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template struct Launch<128, false, true>;
template struct Launch<144, true, true>;
template struct Launch<192, true, true>;
template struct Launch<256, false, true>;
}  // namespace fx
