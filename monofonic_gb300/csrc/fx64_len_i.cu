// Fixed-point transforms of the lengths 112, 150, 180, 324 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template struct Launch<112, false, true>;
template struct Launch<150, true, false>;
template struct Launch<180, true, true>;
template struct Launch<324, true, false>;
}  // namespace fx
