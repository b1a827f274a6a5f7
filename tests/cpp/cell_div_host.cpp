// div_by(v, d, RN(1 / d)) against v / d over the ranges it is used for.
#include "cell_div.h"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

static float bits(uint32_t u) {
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}

int main(int argc, char** argv) {
    const long n = std::atol(argv[1]);
    std::mt19937 rng(5);
    long bad = 0, edge = 0;
    auto check = [&](float v, float d) {
        const float y = 1.0f / d, want = v / d, got = frep::div_by(v, d, y);
        if (std::memcmp(&want, &got, 4) != 0 && bad++ < 5) std::printf("%a / %a: %a, not %a\n", v, d, got, want);
    };
    // a mantissa: random, or one of the ends of its range
    auto mantissa = [&] {
        const uint32_t r = rng();
        if (r & 7) return r >> 9;
        edge++;
        return (r & 8 ? 0x7FFFFFu - (r >> 28) : r >> 28);
    };
    for (long i = 0; i < n; i++) {
        const uint32_t ev = 127 - 100 + rng() % 200, ed = 127 - 20 + rng() % 40;
        check(bits((rng() & 0x80000000u) | ev << 23 | mantissa()), bits(ed << 23 | mantissa()));
    }
    for (float v : {frep::DIV_BY_MIN, frep::DIV_BY_MAX, -frep::DIV_BY_MIN, -frep::DIV_BY_MAX, 1.0f, 2.5f})
        for (float d : {frep::DIV_BY_DMIN, frep::DIV_BY_DMAX, 1.0f, 0.15625f, 2.5f / 12, 2.5f / 240}) check(v, d);
    std::printf("%ld values, %ld edge mantissas, %ld wrong\n", n, edge, bad);
    return bad != 0;
}
