// Power-of-two scales of the fixed-point trainers, from bit patterns.  The differences wrap around, so all of it is unsigned.
#pragma once
#include "layout.cuh"

namespace mascot {

// Bits of 2^(key >> 23) for a key (a difference of two bit patterns) that is not negative, else of 1.
MASCOT_HD constexpr uint32_t scale_bits(int key) { return ((uint32_t)(key > 0 ? key : 0) & 0x7f800000u) + 0x3f800000u; }
// Bits of 1 / s and of 1 / (s t) for powers of two.
MASCOT_HD constexpr uint32_t rev_bits(uint32_t s) { return 0x7f000000u - s; }
MASCOT_HD constexpr uint32_t rev_bits(uint32_t s, uint32_t t) { return 0xbe800000u - s - t; }

}  // namespace mascot
