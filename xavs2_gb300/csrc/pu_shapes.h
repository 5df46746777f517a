// pu_shapes.h -- the 25 PU shapes in LumaPU order (pixel.h:50-65 of the
// reference), for the host.
#pragma once

#include <stdint.h>

namespace xg {

constexpr int kNumParts = 25;
static const uint8_t h_pu_w[kNumParts] = {4, 8, 16, 32, 64, 8, 4, 16, 8, 32, 16, 64, 32,
                                          16, 12, 16, 4, 32, 24, 32, 8, 64, 48, 64, 16};
static const uint8_t h_pu_h[kNumParts] = {4, 8, 16, 32, 64, 4, 8, 8, 16, 16, 32, 32, 64,
                                          12, 16, 4, 16, 24, 32, 8, 32, 48, 64, 16, 64};

}  // namespace xg
