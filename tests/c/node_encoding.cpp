// Rounding of the quantised node planes (bvh8.h): whatever the other half of
// a word holds, a lo plane reads at or below its value and a hi plane at or
// above it, within 2^-6 of the value; the slots word keeps masks and counts.
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "../../cudart_gb300/csrc/bvh8.h"

static float as_float(uint32_t u) {
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}

int main() {
    std::mt19937 rng(1);
    std::uniform_real_distribution<double> unit(0.0, 1.0);
    long checked = 0;
    auto check = [&](double lo, double hi) {
        for (int slot = 0; slot < 8; ++slot) {
            crt::DevNodeQ16 n;
            std::memset(&n, 0xA5, sizeof(n));
            crt::clear_planes16(n);
            crt::set_planes16(n, 1, slot, lo, hi);
            crt::set_planes16(n, 1, slot ^ 4, unit(rng), 1.0 + unit(rng));   // the other half of the same words
            const uint32_t wl = n.planes[1][0][slot & 3], wh = n.planes[1][1][slot & 3];
            const double l = slot < 4 ? as_float(wl << 16) : as_float(wl), h = slot < 4 ? as_float(wh << 16) : as_float(wh);
            // 1e-40: a high half of zero still reads the low half as a denormal
            // (the difference of two floats may lie beyond the largest one: that hi plane reads as
            // infinite or, with a neighbour below it, as NaN, which the slab test's min passes over)
            const bool beyond = hi > (double)FLT_MAX && !std::isfinite(h);
            if (!(l <= lo + 1e-40 && (beyond || h >= hi) && lo - l <= lo * 0x1p-6 + 1e-38 && (beyond || h - hi <= hi * 0x1p-6 + 1e-38))) {
                std::printf("slot %d: [%.17g, %.17g] reads as [%.17g, %.17g]\n", slot, lo, hi, l, h);
                std::exit(1);
            }
            ++checked;
        }
    };
    for (double v : {0.0, 1.0, 1.0 - 0x1p-24, 1.0 + 0x1p-23, 255.0, 256.0, 1.0 / 3.0, 1e-30, 1e30, 0x1p-126, 3e38})
        for (double w : {0.0, 1e-7, 1.0}) check(v, v * (1.0 + w));
    for (int i = 0; i < 200000; ++i) {
        const double lo = std::ldexp(unit(rng), (int)(rng() % 60) - 30);
        check(lo, lo + std::ldexp(unit(rng), (int)(rng() % 60) - 30));
    }
    for (uint32_t mask = 0; mask < 256; ++mask) {
        uint8_t meta[8];
        uint32_t off = 0;
        for (int s = 0; s < 8; ++s) {
            const uint32_t c = (mask * 7u + 3u * s) % 4u;
            meta[s] = (mask >> s) & 1 ? 0x80 : c ? (uint8_t)((c << 5) | off) : 0;
            if (!((mask >> s) & 1)) off += c;
        }
        const uint32_t w = crt::slots_word((uint8_t)mask, meta);
        if ((w & 0xFFu) != mask) return std::printf("mask %u\n", mask), 1;
        for (int s = 0; s < 8; ++s) {
            const uint32_t bits = (w >> (8 + 3 * s)) & 7u, below = (w >> 8) & ((1u << (3 * s)) - 1u);
            const uint32_t want = (mask >> s) & 1 ? 0u : (uint32_t)(meta[s] >> 5);
            if ((uint32_t)__builtin_popcount(bits) != want || (bits & (bits + 1)) != 0) return std::printf("count\n"), 1;
            if (want && (uint32_t)__builtin_popcount(below) != (meta[s] & 31u)) return std::printf("offset\n"), 1;
        }
    }
    std::printf("ok %ld\n", checked);
    return 0;
}
