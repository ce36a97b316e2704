// walknode.h - node records as the ray walk reads them.
//
// A node's reference word (GpuDataStruct word 0) points at its children by the
// grid position of their 2x2x2 block; following it costs the walk an unpack, a
// bounds check and the block-linear index per level.  The pool therefore also
// keeps (memory allowing, nodepool.h) one 8-byte record per node with that index
// worked out when the word is written:
//   x: the resident and constant bits of word 0, and in the low 27 bits the
//      child block (its 8 nodes are 8*block .. 8*block+7), 0 for no children,
//      kLinkBad for a block outside the grid, kLinkOdd for a pointer that is
//      not at a block's corner (its children lie in several blocks: the walk
//      then reads the word itself);
//   y: word 1.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define VV_WALK_HD __host__ __device__ __forceinline__
#else
#define VV_WALK_HD inline
#endif

namespace vv {

constexpr uint32_t kLinkMask = 0x07FFFFFFu, kLinkBad = 0x07FFFFFFu, kLinkOdd = 0x07FFFFFEu;

// Record word x of a node with word 0 in a grid of dx * dy * dz nodes (even, at
// most 1024 per axis, so blocks stay below 2^27 - 2 but for the grid of all
// 1024s, whose last two block numbers read as an odd pointer and go that way).
VV_WALK_HD uint32_t walk_link(uint32_t word0, int dx, int dy, int dz) {
    const uint32_t x = (word0 >> 20) & 0x3FFu, y = (word0 >> 10) & 0x3FFu, z = word0 & 0x3FFu;
    uint32_t link;
    if ((x | y | z) == 0u) {
        link = 0u;
    } else if ((x | y | z) & 1u) {
        link = kLinkOdd;
    } else if (x >= (uint32_t)dx || y >= (uint32_t)dy || z >= (uint32_t)dz) {
        link = kLinkBad;
    } else {
        link = ((z >> 1) * ((uint32_t)dy >> 1) + (y >> 1)) * ((uint32_t)dx >> 1) + (x >> 1);
        if (link > kLinkOdd) link = kLinkOdd;
    }
    return (word0 & 0xC0000000u) | link;
}

// Quotients of block numbers (below 2^27) by a fixed divisor d < 2^19 from one
// multiplication: with 2^l the smallest power of two >= d and
// m = ceil(2^(28+l) / d), m = 2^(28+l)/d + e/d, e < d <= 2^l, so
// n*m / 2^(28+l) exceeds n/d by less than n / (2^28 d) < 1/(2d).
struct BlockDiv {
    uint32_t d, m, l;
};
VV_WALK_HD BlockDiv make_block_div(uint32_t d) {
    BlockDiv b;
    b.d = d;
    b.l = 0u;
    while ((1u << b.l) < d) ++b.l;
    b.m = (uint32_t)((((uint64_t)1 << (28u + b.l)) + d - 1u) / d);
    return b;
}
VV_WALK_HD uint32_t block_div(uint32_t n, const BlockDiv& b) {
#if defined(__CUDA_ARCH__)
    return __umulhi(n << 4, b.m) >> b.l;
#else
    return (uint32_t)(((uint64_t)(n << 4) * b.m) >> 32) >> b.l;
#endif
}

}  // namespace vv
