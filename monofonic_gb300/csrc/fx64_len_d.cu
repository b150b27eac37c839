// Fixed-point transforms of the lengths 576, 768 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template struct Launch<576, true, false>;
template struct Launch<768, true, true>;
}  // namespace fx
