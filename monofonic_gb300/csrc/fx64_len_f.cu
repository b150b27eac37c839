// Fixed-point transforms of the lengths 90, 196, 252, 270 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template struct Launch<90, true, false>;
template struct Launch<196, false, true>;
template struct Launch<252, true, true>;
template struct Launch<270, true, false>;
}  // namespace fx
