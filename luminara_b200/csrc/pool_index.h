// pool_index.h -- place of an item in a warp's pool of paths.
//
// A pool of n slots (pixels) by strata hands out items 0, 1, ...; item idx is slot idx % n of stratum
// idx / n.  The quotient comes from a high multiply where that is exact and from a division elsewhere:
// with magic = ceil(2^32 / n) the product idx * magic exceeds idx * 2^32 / n by less than idx, so its high
// word is idx / n as long as idx * n < 2^32.  Plain C++, so that the rule is checked on the host as well.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define LUM_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define LUM_HOST_DEVICE inline
#endif

namespace lum {

// ceil(2^32 / n) for a pool of n_items items where the high multiply serves all of them; 0: divide.
LUM_HOST_DEVICE uint32_t pool_magic(uint32_t n, uint64_t n_items) {
    return n > 1 && n_items <= (1ull << 32) / n ? 0xFFFFFFFFu / n + 1u : 0u;
}

// idx / n, with the pool's magic.
LUM_HOST_DEVICE uint32_t pool_stratum(uint32_t idx, uint32_t n, uint32_t magic) {
    return magic ? (uint32_t)(((uint64_t)idx * magic) >> 32) : idx / n;
}

}  // namespace lum
