// brick.cuh — the octree levels inside a brick, straight from its occupancy
// bits.
//
// A brick is an aligned cube of 16^3 (dense grids) or 8^3 (mesh folds) cells.
// With its occupancy as one bit per cell in Morton order, a byte of the bits
// is the valid mask of a bottom-level node (bit m for Morton child m, i.e.
// 128 >> i for octant i = 7 - m), the non-zero bytes are the occupancy bits of
// the level above, and so on up to the brick's own node.  So the levels inside
// a brick need no keys, no sorting and no node arrays: per brick, the subtree
// word count and the node's mask go up to the level build, and one pass over
// the bits writes all of the brick's words once its child block's position is
// known.
//
// The words of a brick's subtree are one range, its child block first and
// then each child's subtree in order.  Far pointers never occur inside: the
// range is at most 4096 + 512 + 64 + 8 words, below the 14-bit offset's 16383.
// Let k be the number of the brick's children and n_l(..) count the nodes of
// level l (0: cells, 1: bottom-level nodes) inside the brick in Morton order.
// Relative to the brick's child block, the depth-first order of blocks
// (VoxelOctree.cpp:125-205) puts, for a cell or node in the level-2 node j,
// itself in the level-3 node i in 16^3 bricks,
//     16^3: a cell           k + n_2(through i) + n_1(through j) + n_0(before it)
//           a level-1 node   k + n_2(through i) + n_1(before it) + n_0(before j)
//           a level-2 node   k + n_2(before it) + n_1(before i) + n_0(before i)
//           a level-3 node   its rank among the k
//      8^3: a cell           k + n_1(through j) + n_0(before it)
//           a level-1 node   k + n_1(before it) + n_0(before j)
//           a level-2 node   its rank among the k
// and a node's child block is where its first child is.
#pragma once

#include <cstdint>

namespace svo {

// Coordinates of a cell from its Morton code in the brick (edge at most 16).
__device__ __forceinline__ void brick_cell(uint32_t m, int &x, int &y, int &z) {
    x = (int)((m & 1u) | ((m >> 2) & 2u) | ((m >> 4) & 4u) | ((m >> 6) & 8u));
    y = (int)(((m >> 1) & 1u) | ((m >> 3) & 2u) | ((m >> 5) & 4u) | ((m >> 7) & 8u));
    z = (int)(((m >> 2) & 1u) | ((m >> 4) & 2u) | ((m >> 6) & 4u) | ((m >> 8) & 8u));
}

// The four bits of a 32-cell word's non-zero bytes.
__device__ __forceinline__ uint32_t byte_bits(uint32_t w) {
    w |= w >> 4;
    w |= w >> 2;
    w |= w >> 1;
    w &= 0x01010101u;  // bit 0 of each byte: whether the byte holds a bit
    return (w | (w >> 7) | (w >> 14) | (w >> 21)) & 0xFu;
}

// An 8^3 brick's node from its 16 words of bits, one per lane 0..15 (lanes
// 16..31 hold 0): its mask, and its subtree's words.  All 32 lanes call.
__device__ __forceinline__ void brick8_node(uint32_t w, uint32_t &mask, uint32_t &words) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t other = __shfl_xor_sync(FULL, w, 1);
    const unsigned pairs = __ballot_sync(FULL, (w | other) != 0 && !(lane & 1));
    uint32_t m = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) m |= ((pairs >> (2 * j)) & 1u) << j;
    mask = m;
    const uint32_t n = (uint32_t)__popc(w) + (uint32_t)__popc(byte_bits(w));
    words = __reduce_add_sync(FULL, n) + (uint32_t)__popc(m);
}

}  // namespace svo
