// Fixed-point transforms of the lengths 60, 84, 336, 378 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template struct Launch<60, false, true>;
template struct Launch<84, true, true>;
template struct Launch<336, true, false>;
template struct Launch<378, true, false>;
}  // namespace fx
