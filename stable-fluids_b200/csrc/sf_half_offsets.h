// sf_half_offsets.h -- byte offsets from a cell of one colour to the
// neighbours in the other colour's array (the colour-split layout of the
// red-black solves). They are 32 bits and added modulo 2^32, so a step down is
// the two's complement of the step up: a colour's array is below 4 GB (grids
// below 2^31 cells), but a wrap across it may pass 2^31. Plain C++, so that the
// arithmetic can be checked on the CPU.
#pragma once

#include <cstdint>

#include "sf_types.h"

#ifdef __CUDACC__
#define SFB_HD __host__ __device__ __forceinline__
#else
#define SFB_HD inline
#endif

namespace sfb {

struct HalfOffsets {
    uint32_t plane;       // bytes of a half plane: from z to z + 1
    uint32_t wrap;        // from the bottom plane to the top one (0: no wrap, itself on a face)
    uint32_t y_lo, y_hi;  // rows y - 1 and y + 1 (0 on a face)
    uint32_t x_lo, x_hi;  // cells k0 - 1 and k0 + 4 (on a face a cell of the four)
};

// The thread of cells k0 .. k0 + 3 (of hx a row) in row y; cells of B bytes.
template <int B>
SFB_HD HalfOffsets half_offsets(const Dims& d, int y, int k0, bool px, bool py, bool pz) {
    const uint32_t hx = static_cast<uint32_t>(d.nx) / 2, row = B * hx;
    HalfOffsets o;
    o.plane = row * static_cast<uint32_t>(d.ny);
    o.wrap = pz ? (static_cast<uint32_t>(d.nz) - 1) * o.plane : 0u;
    const uint32_t across = py ? (static_cast<uint32_t>(d.ny) - 1) * row : 0u;
    o.y_lo = y > 0 ? 0u - row : across;
    o.y_hi = y + 1 < d.ny ? row : 0u - across;
    o.x_lo = k0 > 0 ? 0u - B : (px ? row - B : 0u);
    o.x_hi = static_cast<uint32_t>(k0) + 4 < hx ? 4u * B : (px ? 4u * B - row : 3u * B);
    return o;
}

}  // namespace sfb
