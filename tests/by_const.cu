// Host program of test_cells_host.py: by_const against the division.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "cells.cuh"

template <int D>
int check() {
    const float tiny = 1.17549435e-38f;  // smallest normal
    long long bad = 0, ties = 0;
    for (uint64_t b = 0; b <= 0x7f800001ull; b += b >= 0x7f7fff00ull ? 1 : (b < 0x02000000ull ? 7 : 251)) {
        for (uint32_t sign = 0; sign < 2; ++sign) {
            const uint32_t bits = static_cast<uint32_t>(b) | sign << 31;
            float x, got, want;
            std::memcpy(&x, &bits, 4);
            got = wk::by_const<D>(x);
            want = x / D;
            if (std::isnan(want) ? std::isnan(got) : std::memcmp(&got, &want, 4) == 0) continue;
            // the one exception: a tie between subnormal quotients of D = 6
            if (D == 6 && std::fabs(want) < tiny && std::fabs(got - want) <= 1.5e-45f) {
                ++ties;
                continue;
            }
            if (++bad < 4) std::printf("%a / %d: %a, not %a\n", x, D, got, want);
        }
    }
    std::printf("/ %d: %lld wrong, %lld ties\n", D, bad, ties);
    return bad != 0;
}

int main() { return check<3>() | check<6>(); }
