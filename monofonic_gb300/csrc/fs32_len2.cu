// Instances of the single-precision transforms (fs32.cuh): the other grids from
// 56 to 252 with prime factors up to 7 and their padded lengths.
#include "fs32.cuh"

namespace fx {
template struct Launch32<56, false, true>;
template struct Launch32<60, false, true>;
template struct Launch32<72, true, true>;
template struct Launch32<80, false, true>;
template struct Launch32<84, true, true>;
template struct Launch32<90, true, false>;
template struct Launch32<100, false, true>;
template struct Launch32<108, true, true>;
template struct Launch32<112, false, true>;
template struct Launch32<120, true, true>;
template struct Launch32<126, true, false>;
template struct Launch32<140, false, true>;
template struct Launch32<144, true, true>;
template struct Launch32<150, true, false>;
template struct Launch32<160, false, true>;
template struct Launch32<162, true, false>;
}  // namespace fx
