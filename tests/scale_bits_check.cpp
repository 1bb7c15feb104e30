// Host check of csrc/scale_bits.h.  The constants are evaluated at compile time, where an overflow of a signed number is an error.
#include <cmath>
#include <cstdio>
#include <cstring>

#include "scale_bits.h"

using namespace mascot;

constexpr uint32_t one = 0x3f800000u, top60 = one + (60u << 23);
static_assert(rev_bits(one) == one && rev_bits(one, one) == one, "1 / 1");
static_assert(rev_bits(top60, top60) == one - (120u << 23), "1 / 2^120");
static_assert(scale_bits(0) == one && scale_bits(-1) == one && scale_bits(0x3f800000 - 0x7fffffff) == one, "keys that are not positive");
static_assert(scale_bits(0x46ffff00) == 0x86000000u, "the key of a row of zeros (its scale is not used)");

int main() {
    auto of = [](uint32_t b) { float x; std::memcpy(&x, &b, 4); return x; };
    auto bits = [](float x) { uint32_t b; std::memcpy(&b, &x, 4); return b; };
    for (int a = 0; a <= 60; a++) {
        const float s = std::ldexp(1.f, a);
        if (of(scale_bits((a << 23) + 0x123456)) != s || of(rev_bits(bits(s))) != 1.f / s) { std::printf("2^%d\n", a); return 1; }
        for (int b = 0; b <= 60; b++) {
            const float t = std::ldexp(1.f, b);
            if (of(rev_bits(bits(s), bits(t))) != 1.f / (s * t)) { std::printf("2^%d 2^%d\n", a, b); return 1; }
        }
    }
    std::puts("ok");
    return 0;
}
