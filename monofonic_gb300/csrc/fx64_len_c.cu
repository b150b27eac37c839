// Fixed-point transforms of the lengths 288, 384, 512 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template struct Launch<288, true, false>;
template struct Launch<384, true, true>;
template struct Launch<512, false, true>;
}  // namespace fx
