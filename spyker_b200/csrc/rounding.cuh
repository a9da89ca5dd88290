#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

namespace spk
{
// F32(v) > thr, as v > bound: the midpoint between thr and the next float,
// which itself rounds to the even of the two.
inline double rounding_bound(float thr)
{
    if (thr != thr || thr == INFINITY) return INFINITY;
    if (thr == -INFINITY) return -INFINITY;
    const float up = std::nextafterf(thr, INFINITY);
    const double next = std::isinf(up) ? std::ldexp(1.0, 128) : double(up);
    const double mid = double(thr) + (next - double(thr)) * 0.5;
    uint32_t bits;
    std::memcpy(&bits, &thr, 4);
    return bits & 1u ? std::nextafter(mid, -INFINITY) : mid;
}
}  // namespace spk
