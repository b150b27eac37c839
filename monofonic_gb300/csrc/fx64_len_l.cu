// Fixed-point transforms of the lengths 120, 160, 210, 360 (one translation unit per group of
// lengths, compiled in parallel).
#include "fx64_len.cuh"

namespace fx {
template struct Launch<120, true, true>;
template struct Launch<160, false, true>;
template struct Launch<210, true, false>;
template struct Launch<360, true, false>;
}  // namespace fx
