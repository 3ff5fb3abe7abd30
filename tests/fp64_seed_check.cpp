// The reciprocal of fp64_int.cuh from every FP32 seed that the bound of
// rcp.approx (2^-23 of the value) allows. Prints "seeds wrong", exit status 1
// when a reciprocal is not below the true one by less than 8 units of 2^-63.
#include <cmath>
#include <cstdio>
#include <random>

#include "fp64_int.cuh"

int main() {
    std::mt19937_64 gen(11);
    long seeds = 0, wrong = 0;
    auto check = [&](uint64_t D) {
        const uint32_t db = lbm::fi::recip_arg(D);
        float df;
        std::memcpy(&df, &db, 4);
        const double exact = 1.0 / (double)df;
        const unsigned __int128 num = (unsigned __int128)1 << 126;
        const unsigned __int128 want = num / D;  // 1/d, LSB 2^-63, rounded down (2^64 for 1/2)
        float y = (float)exact;
        for (int k = 0; k < 3; k++) y = std::nextafterf(y, 0.0f);
        for (int k = 0; k < 7; k++, y = std::nextafterf(y, 4.0f)) {
            if (std::fabs((double)y - exact) > std::ldexp(exact, -23)) continue;
            uint32_t yb;
            std::memcpy(&yb, &y, 4);
            const uint64_t Y = lbm::fi::recip_refine(D, yb);
            seeds++;
            if ((Y > want || want - Y >= 8) && wrong++ < 5)
                std::printf("D %016llx seed %08x: %016llx, not %016llx\n", (unsigned long long)D, yb,
                            (unsigned long long)Y, (unsigned long long)want);
        }
    };
    const uint64_t one = 1ull << 63, half = 1ull << 62, step = 1ull << 10;  // 53-bit densities
    for (uint64_t q = 0; q < 20000; q++) {
        check(one - step * (q + 1));
        check(half + step * q);
        check(one - (one >> 1) / 20000 * q - step);
    }
    for (int b = 10; b < 62; b++) {
        check(one - (1ull << b));
        check(half + (1ull << b));
    }
    for (int q = 0; q < 1000000; q++) check(half | (gen() >> 2 & ~(step - 1)));
    std::printf("%ld %ld\n", seeds, wrong);
    return wrong != 0;
}
