// Fixed-point transforms of the length 1152 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template struct Launch<1152, true, false>;
}  // namespace fx
