// Instances of the single-precision transforms (fs32.cuh): padded lengths and
// grid lengths of powers of two, and grid lengths of the fused transforms.
#include "fs32.cuh"

namespace fx {
template struct Launch32<16, false, true>;
template struct Launch32<24, true, true>;
template struct Launch32<32, false, true>;
template struct Launch32<48, true, true>;
template struct Launch32<64, false, true>;
template struct Launch32<96, true, true>;
template struct Launch32<128, false, true>;
template struct Launch32<192, true, true>;
template struct Launch32<256, false, true>;
template struct Launch32<384, true, true>;
template struct Launch32<512, false, true>;
template struct Launch32<768, true, true>;
}  // namespace fx
