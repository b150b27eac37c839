// Fixed-point transforms of the lengths 140, 200, 224, 240, 294 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template struct Launch<140, false, true>;
template struct Launch<200, false, true>;
template struct Launch<224, false, true>;
template struct Launch<240, true, true>;
template struct Launch<294, true, false>;
}  // namespace fx
