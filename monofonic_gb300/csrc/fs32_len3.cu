// Instances of the single-precision transforms (fs32.cuh): the other grids from
// 56 to 252 with prime factors up to 7 and their padded lengths.
#include "fs32.cuh"

namespace fx {
template struct Launch32<168, true, true>;
template struct Launch32<180, true, true>;
template struct Launch32<196, false, true>;
template struct Launch32<200, false, true>;
template struct Launch32<210, true, false>;
template struct Launch32<216, true, true>;
template struct Launch32<224, false, true>;
template struct Launch32<240, true, true>;
template struct Launch32<252, true, true>;
template struct Launch32<270, true, false>;
template struct Launch32<294, true, false>;
template struct Launch32<300, true, false>;
template struct Launch32<324, true, false>;
template struct Launch32<336, true, false>;
template struct Launch32<360, true, false>;
template struct Launch32<378, true, false>;
}  // namespace fx
