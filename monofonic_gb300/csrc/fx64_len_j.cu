// Fixed-point transforms of the lengths 100, 108, 162, 168 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template struct Launch<100, false, true>;
template struct Launch<108, true, true>;
template struct Launch<162, true, false>;
template struct Launch<168, true, true>;
}  // namespace fx
