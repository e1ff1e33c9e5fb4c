// Sums of counts that stop at a ceiling instead of wrapping round: the lengths
// of the raster's tile lists (raster.cuh), whose sum passes 2^32 where a
// caller's grid makes tens of millions of triangles that each meet hundreds of
// tiles.  Such a sum does not depend on the order of its terms.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define IDL_HOST_DEVICE __host__ __device__
#else
#define IDL_HOST_DEVICE
#endif

namespace idl {

constexpr int32_t SUM_CEILING = 0x7FFFFFFF;

// a, b >= 0
IDL_HOST_DEVICE inline int32_t held_sum(int32_t a, int32_t b)
{
    const uint32_t s = (uint32_t)a + (uint32_t)b;   // below 2^32
    return s < (uint32_t)SUM_CEILING ? (int32_t)s : SUM_CEILING;
}

}  // namespace idl
