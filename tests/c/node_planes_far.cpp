// Lo planes further from their node's origin than the largest float (the
// origin and the plane at opposite ends of the range): whatever the other half of
// the word holds, the plane reads as a number at or below its value.
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "../../cudart_gb300/csrc/bvh8.h"

int main() {
    const double top = (double)FLT_MAX;
    for (double v : {0x1p127, top * (1 - 0x1p-9), top, top * (1 + 0x1p-26), top * (1 + 0x1p-24), top * 1.25, top * 2})
        for (double other : {0.0, 1e-39, 0.75, 3.0, top, 2 * top})
            for (int slot = 0; slot < 8; ++slot) {
                crt::DevNodeQ16 n;
                crt::clear_planes16(n);
                crt::set_planes16(n, 2, slot ^ 4, other, other);
                crt::set_planes16(n, 2, slot, v, v);
                uint32_t w = n.planes[2][0][slot & 3];
                if (slot < 4) w <<= 16;
                float f;
                std::memcpy(&f, &w, 4);
                if (!(std::isfinite(f) && (double)f <= v && (double)f >= 0x1p126))
                    return std::printf("slot %d: %.9g beside %.9g reads as %.9g\n", slot, v, other, f), 1;
            }
    std::printf("ok\n");
    return 0;
}
