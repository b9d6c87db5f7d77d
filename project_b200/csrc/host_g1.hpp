// Sums of points on the host: chains that are serial whatever they run on (an Fp multiplication takes about 80 ns
// there and 1 us as the only work of a warp).
#pragma once

#include <cstdint>
#include <cstring>

#include "g1.cuh"

namespace gzk
{
    // sum_w 2^(c w) points[w], `count` > 0 of them
    inline G1Xyzz host_horner(const G1Xyzz* points, size_t count, unsigned c)
    {
        G1Xyzz acc = points[count - 1];
        for (size_t w = count - 1; w-- > 0;)
        {
            for (unsigned k = 0; k < c; ++k) acc = g1_double(acc);
            acc = g1_add(acc, points[w]);
        }
        return acc;
    }

    // Canonical affine coordinates in wire format (96 zero bytes for the point at infinity)
    inline void host_to_affine_bytes(const G1Xyzz& p, uint8_t out[96])
    {
        const G1Affine a = g1_to_affine(p);
        const Fp x = from_mont(a.x), y = from_mont(a.y);
        std::memcpy(out, x.l, 48);
        std::memcpy(out + 48, y.l, 48);
    }
}
