// Fixed-point transforms of the lengths 56, 80, 126, 216, 300 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template struct Launch<56, false, true>;
template struct Launch<80, false, true>;
template struct Launch<126, true, false>;
template struct Launch<216, true, true>;
template struct Launch<300, true, false>;
}  // namespace fx
