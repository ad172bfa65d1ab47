// build.cu — GPU octree construction from a dense voxel grid.
//
// Replaces VoxelOctree(VoxelData*) (VoxelOctree.cpp:125-205) with its
// ChunkedAllocator far-pointer splice (ChunkedAllocator.hpp:76-114).  The
// reference builds depth first and patches far pointers afterwards; this
// pipeline computes the same word stream in three data-parallel phases.
// Voxels that come as bricks (a dense grid's, a mesh fold's) take a shorter
// way to the same words, over the bricks' occupancy bits and a dense pyramid
// above them (brick.cuh, build_pyramid); the phases serve streamed files,
// cache blocks smaller than a brick and, from phase 2 on, the bricks of cubes
// too large for the pyramid:
//
//  1. Extraction.  The grid is read brick by brick (16^3 voxels per CTA,
//     bricks visited in Morton order) and occupied voxels are emitted as
//     (Morton key, payload) pairs in global Morton order.  Child slots in the
//     reference are in descending octant index i, and octant i = 7 - m where
//     m = xbit | ybit<<1 | zbit<<2 (VoxelOctree.cpp:144-146), so ascending
//     Morton order is exactly the reference's depth-first child order.
//  2. Bottom-up levels.  Children are grouped by key>>3 (head flags + scan);
//     each parent gets its valid mask (bit m for child m, i.e. 128>>i) and,
//     from its children's subtree word counts S, the far-pointer decision of
//     VoxelOctree.cpp:172-183: offset_i = (k-i) + sum_{j<i} S_j and the
//     parent's children carry far words when any offset_i > 0x3FFF.
//     S = k*(far ? 2 : 1) + sum_j S_j (k payload words at the bottom level).
//  3. Top-down placement.  Root at 0 with its child block at 1; a parent with
//     block start B puts child i at B + i*stride and child i's block at
//     B + k*stride + sum_{j<i} S_j, then writes the child's descriptor with
//     offset = block - position (plus k-i far words, VoxelOctree.cpp:190-191)
//     and, when far, the low 32 bits in the next word.
//
// VoxelData corner cases (VoxelData.cpp:160-175, 120-158, 211-262) that the
// reference's output depends on, for cache-block edge M chosen from `mem`:
//   - with M >= 4 and odd data depth the last z slice never reaches the
//     low-level lookup table, so its voxels are dropped;
//   - nodes of edge >= M come from the top lookup table, which is built from
//     the full data, so an M-block whose only voxels lie in that slice still
//     appears as a descriptor with no children.
#include <cstdio>
#include <mutex>

#include "brick.cuh"
#include "chain.cuh"
#include "morton.cuh"
#include "scan.cuh"
#include "svo_internal.h"

namespace svo {
namespace {

constexpr int kBrickThreads = 256;

struct GridGeom {
    const uint32_t *grid;
    int w, h, d;
    int log_brick;      // brick edge E = 1 << log_brick
    int drop_last_z;    // 1: voxels at z == d-1 are excluded from the output
    int log_block;      // cache-block edge M = 1 << log_block
    uint8_t *topflag;   // per M-block "has any voxel" (Morton-indexed), or null
};

// Whether the grid's rows start on 16-byte boundaries, so that a uint4 of a
// 16^3 brick lies wholly inside the grid or outside.
__device__ __forceinline__ bool grid_vec4(const GridGeom &g) {
    return (g.w & 3) == 0 && (reinterpret_cast<uintptr_t>(g.grid) & 15) == 0;
}

// A 16^3 brick wholly inside the grid, whose rows start on 16-byte
// boundaries, is read as 1024 uint4 (4 per thread of a 256-thread CTA).
// uint4 q of the brick covers x = 4*(q & 3) .. +3, y = (q >> 2) & 15,
// z = q >> 6, i.e. cells 4q .. 4q+3 of the brick's row-major order.
__device__ __forceinline__ bool brick_vec4(const GridGeom &g, int gx0, int gy0, int gz0) {
    return g.log_brick == 4 && kBrickThreads == 256 && gx0 + 16 <= g.w && gy0 + 16 <= g.h && gz0 + 16 <= g.d &&
           (g.w & 3) == 0 && (reinterpret_cast<uintptr_t>(g.grid) & 15) == 0;
}

// Loads the brick's 4 uint4 of this thread, all issued before any is used:
// a scan of the whole grid is bound by the loads in flight, not by the
// instructions that test them.
__device__ __forceinline__ void brick_load4(const GridGeom &g, int gx0, int gy0, int gz0, uint4 (&v)[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int q = threadIdx.x + k * 256;
        const int gx = gx0 + ((q & 3) << 2), gy = gy0 + ((q >> 2) & 15), gz = gz0 + (q >> 6);
        v[k] = __ldg(reinterpret_cast<const uint4 *>(g.grid + (uint64_t)gx +
                                                     (uint64_t)g.w * ((uint64_t)gy + (uint64_t)g.h * gz)));
    }
}

// Phase 1a: per brick, count voxels that survive (V') and flag M-blocks that
// hold any voxel (V).  One CTA per brick; consecutive threads read
// consecutive x so each warp load covers whole 32-byte sectors of a row.
__global__ void __launch_bounds__(kBrickThreads, 8) k_brick_count(GridGeom g, uint64_t n_bricks, uint32_t *__restrict__ counts) {
    const int lb = g.log_brick;
    const int E = 1 << lb;
    const int cells = E * E * E;
    for (uint64_t b = blockIdx.x; b < n_bricks; b += gridDim.x) {
        uint32_t bx = compact3(b), by = compact3(b >> 1), bz = compact3(b >> 2);
        int gx0 = (int)(bx << lb), gy0 = (int)(by << lb), gz0 = (int)(bz << lb);
        uint32_t cnt = 0, any = 0;
        if (brick_vec4(g, gx0, gy0, gz0)) {
            uint4 v[4];
            brick_load4(g, gx0, gy0, gz0, v);
            if (!(g.topflag && g.log_block < lb)) {
                // no cell-level flags: count the row's nonzero words and OR
                // them for the brick's flag (a scan of the grid is otherwise
                // bound by these instructions, not by its loads)
                uint32_t bits = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int gz = gz0 + ((threadIdx.x + k * 256) >> 6);
                    bits |= v[k].x | v[k].y | v[k].z | v[k].w;
                    const uint32_t nz = (uint32_t)(v[k].x != 0u) + (uint32_t)(v[k].y != 0u) +
                                        (uint32_t)(v[k].z != 0u) + (uint32_t)(v[k].w != 0u);
                    if (!(g.drop_last_z && gz == g.d - 1)) cnt += nz;
                }
                any = bits != 0u;
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int q = threadIdx.x + k * 256;
                    const int gx = gx0 + ((q & 3) << 2), gy = gy0 + ((q >> 2) & 15), gz = gz0 + (q >> 6);
                    const uint32_t e[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (e[j]) {
                            any = 1;
                            if (!(g.drop_last_z && gz == g.d - 1)) ++cnt;
                            g.topflag[morton3((uint32_t)(gx + j) >> g.log_block, (uint32_t)gy >> g.log_block,
                                              (uint32_t)gz >> g.log_block)] = 1;
                        }
                    }
                }
            }
        } else if (gx0 < g.w && gy0 < g.h && gz0 < g.d) {
            for (int c = threadIdx.x; c < cells; c += kBrickThreads) {
                int gx = gx0 + (c & (E - 1)), gy = gy0 + ((c >> lb) & (E - 1)), gz = gz0 + (c >> (2 * lb));
                if (gx < g.w && gy < g.h && gz < g.d) {
                    uint32_t v = __ldg(g.grid + (uint64_t)gx + (uint64_t)g.w * ((uint64_t)gy + (uint64_t)g.h * gz));
                    if (v) {
                        any = 1;
                        if (!(g.drop_last_z && gz == g.d - 1)) ++cnt;
                        if (g.topflag && g.log_block < lb)
                            g.topflag[morton3((uint32_t)gx >> g.log_block, (uint32_t)gy >> g.log_block,
                                              (uint32_t)gz >> g.log_block)] = 1;
                    }
                }
            }
        }
        uint32_t total;
        block_excl_scan<uint32_t>(cnt, &total);
        int block_any = __syncthreads_or(any);
        if (threadIdx.x == 0) {
            counts[b] = total;
            if (block_any && g.topflag && g.log_block >= lb)
                g.topflag[b >> (3 * (g.log_block - lb))] = 1;
        }
    }
}

// Phase 1b: emit (key, payload) for V' in Morton order.  The brick goes into
// shared memory in local Morton order as it is read (a thread's uint4 holds
// cells x .. x+3 of a row, whose codes are m, m+1, m+8 and m+9 with m the
// code of x), so nothing is decoded afterwards.  Warp w then owns codes
// [w * span, (w + 1) * span): one pass counts its occupied cells with
// ballots, and after the warps' totals are known, a second pass writes their
// keys and payloads at consecutive positions.
__global__ void __launch_bounds__(kBrickThreads) k_brick_emit(GridGeom g, uint64_t n_bricks, const uint32_t *__restrict__ counts,
                                                            const uint64_t *__restrict__ offsets,
                                                            uint64_t *__restrict__ keys, uint32_t *__restrict__ payload) {
    constexpr int kWarps = kBrickThreads / 32;
    __shared__ __align__(16) uint32_t tile[16 * 16 * 16];  // the brick's words by local Morton code
    __shared__ uint32_t wtot[kWarps];
    const int lb = g.log_brick;
    const int E = 1 << lb;
    const int cells = E * E * E;
    const int span = (cells + kWarps - 1) / kWarps;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const int m_lo = wid * span, m_hi = min(cells, m_lo + span);
    for (uint64_t b = blockIdx.x; b < n_bricks; b += gridDim.x) {
        if (counts[b] == 0) continue;  // uniform across the CTA
        uint32_t bx = compact3(b), by = compact3(b >> 1), bz = compact3(b >> 2);
        int gx0 = (int)(bx << lb), gy0 = (int)(by << lb), gz0 = (int)(bz << lb);
        if (brick_vec4(g, gx0, gy0, gz0)) {
            uint4 v[4];
            brick_load4(g, gx0, gy0, gz0, v);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int q = threadIdx.x + k * 256;
                if (g.drop_last_z && gz0 + (q >> 6) == g.d - 1) v[k] = make_uint4(0u, 0u, 0u, 0u);
                const uint32_t m = (uint32_t)morton3((uint32_t)((q & 3) << 2), (uint32_t)((q >> 2) & 15),
                                                     (uint32_t)(q >> 6));
                tile[m] = v[k].x;
                tile[m + 1] = v[k].y;
                tile[m + 8] = v[k].z;
                tile[m + 9] = v[k].w;
            }
        } else {
            for (int c = threadIdx.x; c < cells; c += kBrickThreads) {
                int lx = c & (E - 1), ly = (c >> lb) & (E - 1), lz = c >> (2 * lb);
                int gx = gx0 + lx, gy = gy0 + ly, gz = gz0 + lz;
                uint32_t v = 0;
                if (gx < g.w && gy < g.h && gz < g.d && !(g.drop_last_z && gz == g.d - 1))
                    v = __ldg(g.grid + (uint64_t)gx + (uint64_t)g.w * ((uint64_t)gy + (uint64_t)g.h * gz));
                tile[morton3((uint32_t)lx, (uint32_t)ly, (uint32_t)lz)] = v;
            }
        }
        __syncthreads();
        uint32_t run = 0;
        for (int m0 = m_lo; m0 < m_hi; m0 += 32) {
            const int m = m0 + lane;
            run += (uint32_t)__popc(__ballot_sync(0xffffffffu, m < m_hi && tile[m] != 0u));
        }
        if (lane == 0) wtot[wid] = run;
        __syncthreads();
        uint64_t out = offsets[b];
        for (int w = 0; w < wid; ++w) out += wtot[w];
        const uint64_t kbase = b << (3 * lb);
        for (int m0 = m_lo; m0 < m_hi; m0 += 32) {
            const int m = m0 + lane;
            const uint32_t v = m < m_hi ? tile[m] : 0u;
            const uint32_t ball = __ballot_sync(0xffffffffu, v != 0u);
            if (v) {
                const uint64_t o = out + (uint64_t)__popc(ball & lt);
                keys[o] = kbase | (uint64_t)m;
                payload[o] = v;
            }
            out += (uint64_t)__popc(ball);
        }
        __syncthreads();  // the next brick overwrites tile and wtot
    }
}

// The sum of a tile array before `tile`, by the whole CTA: with up to
// kSelfScanTiles tiles this replaces a scan launch.
constexpr uint64_t kSelfScanTiles = 1024;

__device__ __forceinline__ uint32_t tiles_before(const uint32_t *__restrict__ tile_n, uint32_t tile) {
    uint32_t n = 0;
    for (uint32_t t = threadIdx.x; t < tile; t += blockDim.x) n += __ldg(tile_n + t);
    uint32_t total;
    block_excl_scan<uint32_t>(n, &total);
    return total;
}

// ---- bricks of 16^3 cells, straight to the words -------------------------------

// Row-major index, among the 16^3 bricks that cover the grid, of the one at
// (gx0, gy0, gz0): where its bits are.  (The Morton codes run over the whole
// cube, which a thin grid fills only in a small part.)
__device__ __forceinline__ uint64_t brick_linear(const GridGeom &g, int gx0, int gy0, int gz0) {
    return (uint64_t)(gx0 >> 4) +
           (uint64_t)((g.w + 15) >> 4) * ((uint64_t)(gy0 >> 4) + (uint64_t)((g.h + 15) >> 4) * (uint64_t)(gz0 >> 4));
}

// Phase 1 of the brick build: per brick its occupancy bits (128 words by
// Morton code, written for bricks that hold a voxel), its node's mask and
// subtree words (0 for an empty brick), and the cache blocks' flags.  A lane's
// uint4 gives 4 bits of the 32-cell word that its x/4 column shares with 7
// other lanes, so three shuffles OR the word together and no atomics are
// needed.  Reads the grid once: bound by HBM, 87 us for the 512^3 cells of a
// sphere union (0.54 GB at 6.2 TB/s).  6 CTAs of 42 registers per SM: at 8 the
// word-by-word branch spills.
// any_of: optionally, whether a brick holds a voxel at all, dropped slice
// included; list, n_list: optionally, the bricks with surviving voxels, in any
// order; n_voxels: optionally, those voxels' total.
__global__ void __launch_bounds__(kBrickThreads, 6) k_brick_bits(GridGeom g, uint64_t n_bricks,
                                                                 uint32_t *__restrict__ bits,
                                                                 uint32_t *__restrict__ words_of,
                                                                 uint8_t *__restrict__ mask_of,
                                                                 uint8_t *__restrict__ any_of,
                                                                 uint32_t *__restrict__ list,
                                                                 uint32_t *__restrict__ n_list,
                                                                 unsigned long long *__restrict__ n_voxels) {
    // Alternating: warp 0 may still read the brick before.  Every brick that
    // takes a buffer passes a barrier after writing it, so the bits written to
    // a buffer follow, by the barrier of the brick between, the reads of its
    // last use.
    __shared__ __align__(16) uint32_t sbits[2][128];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int turn = 0;
    const int x4 = lane & 3, yl = (lane >> 2) & 3, zl = lane >> 4;
    const bool vec4 = grid_vec4(g);
    for (uint64_t b = blockIdx.x; b < n_bricks; b += gridDim.x) {
        const int gx0 = (int)(compact3(b) << 4), gy0 = (int)(compact3(b >> 1) << 4), gz0 = (int)(compact3(b >> 2) << 4);
        uint32_t any = 0;
        const bool inside = gx0 < g.w && gy0 < g.h && gz0 < g.d;  // else the cube's padding
        uint32_t *const sb = sbits[turn];
        if (inside) turn ^= 1;
        if (!inside) {
            // no barrier is passed here, so the buffer stays for the next brick
        } else if (vec4) {
            // warp w takes the columns (y / 4, z / 2) = w, w + 8, w + 16, w + 24
            uint4 v[4];
            const int gx = gx0 + 4 * x4, gy = gy0 + 4 * (wid & 3) + yl, gz = gz0 + 2 * (wid >> 2) + zl;
            const uint32_t *const at = g.grid + (uint64_t)gx + (uint64_t)g.w * ((uint64_t)gy + (uint64_t)g.h * gz);
            const bool row = gx < g.w && gy < g.h;
#pragma unroll
            for (int k = 0; k < 4; ++k)  // wid + 8 k: the same y, z + 4 k
                v[k] = row && gz + 4 * k < g.d ? __ldg(reinterpret_cast<const uint4 *>(at + (uint64_t)(4 * k) * g.w * g.h))
                                               : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int k = 0; k < 4; ++k) any |= v[k].x | v[k].y | v[k].z | v[k].w;
            any = (uint32_t)__syncthreads_or((int)(any != 0));
            if (any) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int c = wid + 8 * k, y4 = c & 3, z2 = c >> 2;
                    uint32_t w = (uint32_t)(v[k].x != 0u) | ((uint32_t)(v[k].y != 0u) << 1) |
                                 ((uint32_t)(v[k].z != 0u) << 8) | ((uint32_t)(v[k].w != 0u) << 9);
                    w <<= ((yl & 1) << 1) | ((yl >> 1) << 4) | (zl << 2);
                    if (g.drop_last_z && gz0 + 2 * z2 + zl == g.d - 1) w = 0;
                    w |= __shfl_xor_sync(FULL, w, 4);
                    w |= __shfl_xor_sync(FULL, w, 8);
                    w |= __shfl_xor_sync(FULL, w, 16);
                    if (lane < 4)
                        sb[(z2 & 1) | ((x4 & 1) << 1) | ((y4 & 1) << 2) | (((z2 >> 1) & 1) << 3) | ((x4 >> 1) << 4) |
                           ((y4 >> 1) << 5) | ((z2 >> 2) << 6)] = w;
                }
            }
        } else {
            // a lane per cell of a 32-cell word: the ballot is the word
            for (int h = 0; h < 16; h += 4) {
                uint32_t v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    int x, y, z;
                    brick_cell((uint32_t)((wid * 16 + h + k) * 32 + lane), x, y, z);
                    const int gx = gx0 + x, gy = gy0 + y, gz = gz0 + z;
                    v[k] = gx < g.w && gy < g.h && gz < g.d
                               ? __ldg(g.grid + (uint64_t)gx + (uint64_t)g.w * ((uint64_t)gy + (uint64_t)g.h * gz))
                               : 0u;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    int x, y, z;
                    brick_cell((uint32_t)((wid * 16 + h + k) * 32 + lane), x, y, z);
                    any |= v[k];
                    const uint32_t w = __ballot_sync(FULL, v[k] != 0u && !(g.drop_last_z && gz0 + z == g.d - 1));
                    if (lane == 0) sb[wid * 16 + h + k] = w;
                }
            }
            any = (uint32_t)__syncthreads_or((int)(any != 0));
        }
        if (!any) {
            if (threadIdx.x == 0) {
                words_of[b] = 0;
                mask_of[b] = 0;
                if (any_of) any_of[b] = 0;
            }
            continue;
        }
        __syncthreads();
        if (wid == 0) {
            const uint4 w = reinterpret_cast<const uint4 *>(sb)[lane];
            reinterpret_cast<uint4 *>(bits + brick_linear(g, gx0, gy0, gz0) * 128)[lane] = w;
            const uint32_t n0 = (uint32_t)(__popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w));
            const uint32_t n1 = (uint32_t)(__popc(byte_bits(w.x)) + __popc(byte_bits(w.y)) + __popc(byte_bits(w.z)) +
                                           __popc(byte_bits(w.w)));
            const uint32_t n2 = (uint32_t)((w.x | w.y) != 0u) + (uint32_t)((w.z | w.w) != 0u);
            const unsigned full = __ballot_sync(FULL, n2 != 0);
            uint32_t mask = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) mask |= (uint32_t)(((full >> (4 * i)) & 15u) != 0) << i;
            const uint32_t total = __reduce_add_sync(FULL, n0 + n1 + n2), cells = __reduce_add_sync(FULL, n0);
            if (lane == 0) {
                words_of[b] = total + (uint32_t)__popc(mask);
                mask_of[b] = (uint8_t)mask;
                if (any_of) any_of[b] = 1;
                if (g.topflag) g.topflag[b >> (3 * (g.log_block - 4))] = 1;
                if (list && cells) list[atomicAdd(n_list, 1u)] = (uint32_t)b;
                if (n_voxels && cells) atomicAdd(n_voxels, (unsigned long long)cells);
            }
        }
    }
}

// Where the bricks that hold something are: their keys (the brick's Morton
// code; key_of[j] where given, else j), masks and subtree words move to
// consecutive entries, with the brick's own index in src.
struct BrickNodes {
    uint64_t n;                   // bricks
    const uint32_t *key_of;       // or null
    const uint32_t *words_of;
    const uint8_t *mask_of;
    const uint8_t *any_of;        // or null: a brick is kept when it has words
};

constexpr int kNodeItems = 8, kNodeTile = kBrickThreads * kNodeItems;

__device__ __forceinline__ bool brick_kept(const BrickNodes &b, uint64_t j) {
    return j < b.n && (b.any_of ? b.any_of[j] != 0 : b.words_of[j] != 0u);
}

// Thread t of a tile looks at bricks 8t .. 8t + 7.
__global__ void __launch_bounds__(kBrickThreads) k_brick_keep_count(BrickNodes b, uint32_t *__restrict__ tile_n) {
    const uint64_t j0 = (uint64_t)blockIdx.x * kNodeTile + (uint64_t)threadIdx.x * kNodeItems;
    uint32_t n = 0;
#pragma unroll
    for (int k = 0; k < kNodeItems; ++k) n += brick_kept(b, j0 + k) ? 1u : 0u;
    uint32_t total;
    block_excl_scan<uint32_t>(n, &total);
    if (threadIdx.x == 0) tile_n[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kBrickThreads) k_brick_keep(BrickNodes b, const uint32_t *__restrict__ tile_n,
                                                              const uint32_t *__restrict__ tile_first,
                                                              uint64_t *__restrict__ key, uint32_t *__restrict__ src,
                                                              uint8_t *__restrict__ mask, uint8_t *__restrict__ count,
                                                              uint64_t *__restrict__ S, uint32_t *__restrict__ n_kept) {
    const uint32_t first = tile_first ? tile_first[blockIdx.x] : tiles_before(tile_n, blockIdx.x);
    const uint64_t j0 = (uint64_t)blockIdx.x * kNodeTile + (uint64_t)threadIdx.x * kNodeItems;
    uint32_t n = 0, keep = 0;
#pragma unroll
    for (int k = 0; k < kNodeItems; ++k)
        if (brick_kept(b, j0 + k)) {
            keep |= 1u << k;
            ++n;
        }
    uint32_t total;
    uint32_t o = first + block_excl_scan<uint32_t>(n, &total);
    for (; keep; keep &= keep - 1, ++o) {
        const uint64_t j = j0 + (uint64_t)(__ffs((int)keep) - 1);
        key[o] = b.key_of ? (uint64_t)b.key_of[j] : j;
        src[o] = (uint32_t)j;
        mask[o] = b.mask_of[j];
        count[o] = (uint8_t)__popc((uint32_t)b.mask_of[j]);
        S[o] = b.words_of[j];
    }
    if (!tile_first && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *n_kept = first + total;
}

// The bricks to place: n of them, with subtree words and child block position
// indexed by the brick (dense: words_of, B) or by its entry among the kept
// nodes (S, B, their keys in key), src holding the bricks (dense) or, for 8^3
// bricks, the index of their bits and voxels.
struct BrickPlaces {
    const uint32_t *n;
    const uint32_t *src;
    const uint64_t *key;
    const uint32_t *words_of;
    const uint64_t *S, *B;
};

template <bool kDense>
__device__ __forceinline__ void brick_place(const BrickPlaces &a, uint64_t p, uint64_t &b, uint64_t &at, uint64_t &size) {
    if (kDense) {
        b = a.src[p];
        at = a.B[b];
        size = a.words_of[b];
    } else {
        b = a.key[p];
        at = a.B[p];
        size = a.S[p];
    }
}

// The last phase of the brick build: every brick's words, relative to its
// child block (brick.cuh gives the positions).  The 32 lanes of
// the first warp scan the level counts, four 32-cell words each; 128 threads
// write the bottom-level nodes, and the warps copy the voxels, in Morton order
// with consecutive lanes on consecutive cells.  A range past the word count is
// reported through *err and not written.
//
// Bound by memory: it reads the occupied bricks again and writes the words.  A
// 512^3 grid's (42 M words): 53 us with six CTAs an SM and all of a brick's
// reads under way before its place is looked at, 56 with four CTAs, 59 with
// the cells read after the place.
template <bool kDense>
__global__ void __launch_bounds__(kBrickThreads, 6) k_place_brick16(GridGeom g, BrickPlaces at_of,
                                                                 const uint32_t *bits,
                                                                 uint32_t *__restrict__ words, uint64_t W,
                                                                 uint32_t *__restrict__ err) {
    chain_begin();
    __shared__ __align__(16) uint32_t tile[16 * 16 * 16];  // a whole brick's words by Morton code
    __shared__ __align__(16) uint32_t sb[128];
    __shared__ uint16_t cell_at[128];  // per 32-cell word: where its cells go
    __shared__ uint16_t node_at[128];  // ... and its bottom-level nodes
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const bool vec = grid_vec4(g);
    const uint32_t n = *at_of.n;
    for (uint32_t p = blockIdx.x; p < n; p += gridDim.x) {
        // the place, the cells and the bits are all on their way before the
        // place is looked at
        uint64_t b, at, size;
        brick_place<kDense>(at_of, p, b, at, size);
        const int gx0 = (int)(compact3(b) << 4), gy0 = (int)(compact3(b >> 1) << 4), gz0 = (int)(compact3(b >> 2) << 4);
        uint4 v[4], own_bits = make_uint4(0u, 0u, 0u, 0u);
        if (vec) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int q = threadIdx.x + k * 256;
                const int gx = gx0 + ((q & 3) << 2), gy = gy0 + ((q >> 2) & 15), gz = gz0 + (q >> 6);
                v[k] = gx < g.w && gy < g.h && gz < g.d
                           ? __ldg(reinterpret_cast<const uint4 *>(
                                 g.grid + (uint64_t)gx + (uint64_t)g.w * ((uint64_t)gy + (uint64_t)g.h * gz)))
                           : make_uint4(0u, 0u, 0u, 0u);
            }
        }
        if (wid == 0) own_bits = __ldg(reinterpret_cast<const uint4 *>(bits + brick_linear(g, gx0, gy0, gz0) * 128) + lane);
        if (size == 0) continue;  // only a dropped slice's voxels: no children
        if (at + size > W) {
            if (threadIdx.x == 0) atomicOr(err, 4u);
            continue;
        }
        uint32_t *const out = words + at;
        __syncthreads();  // the previous brick's readers are done
        if (wid == 0) {
            const uint4 w = own_bits;
            reinterpret_cast<uint4 *>(sb)[lane] = w;
            const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
            uint32_t c0 = 0, c1 = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                c0 += (uint32_t)__popc(ww[k]);
                c1 += (uint32_t)__popc(byte_bits(ww[k]));
            }
            const uint32_t ja = (w.x | w.y) != 0u, jb = (w.z | w.w) != 0u;
            // cells in bits 0..12, bottom-level nodes in 13..22, level-2 nodes in 23..29
            const uint32_t own = c0 | (c1 << 13) | ((ja + jb) << 23);
            const uint32_t incl = warp_incl_scan(own), excl = incl - own;
            const unsigned full = __ballot_sync(FULL, (ja | jb) != 0u);
            uint32_t mask = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) mask |= (uint32_t)(((full >> (4 * i)) & 15u) != 0) << i;
            const uint32_t k3 = (uint32_t)__popc(mask);
            // the level-3 node of this lane is lanes 4i .. 4i + 3
            const uint32_t bi = __shfl_sync(FULL, excl, lane & ~3), ti = __shfl_sync(FULL, incl, lane | 3);
            const uint32_t n2t = ti >> 23;
            const uint32_t n0 = excl & 0x1FFFu, n1 = (excl >> 13) & 0x3FFu, n2 = excl >> 23;
            const uint32_t m1[4] = {byte_bits(w.x), byte_bits(w.y), byte_bits(w.z), byte_bits(w.w)};
            const uint32_t a1 = (uint32_t)__popc(m1[0] | (m1[1] << 4)), p0 = (uint32_t)__popc(w.x);
            const uint32_t p1 = (uint32_t)__popc(w.y), p2 = (uint32_t)__popc(w.z), a0 = p0 + p1;
            const uint32_t base = k3 + n2t;
            cell_at[4 * lane] = (uint16_t)(base + n1 + a1 + n0);
            cell_at[4 * lane + 1] = (uint16_t)(base + n1 + a1 + n0 + p0);
            cell_at[4 * lane + 2] = (uint16_t)(base + n1 + c1 + n0 + a0);
            cell_at[4 * lane + 3] = (uint16_t)(base + n1 + c1 + n0 + a0 + p2);
            node_at[4 * lane] = (uint16_t)(base + n1 + n0);
            node_at[4 * lane + 1] = (uint16_t)(base + n1 + (uint32_t)__popc(m1[0]) + n0);
            node_at[4 * lane + 2] = (uint16_t)(base + n1 + a1 + n0 + a0);
            node_at[4 * lane + 3] = (uint16_t)(base + n1 + a1 + (uint32_t)__popc(m1[2]) + n0 + a0);
            // level-2 nodes 2 lane and 2 lane + 1
            const uint32_t before_i = ((bi >> 13) & 0x3FFu) + (bi & 0x1FFFu);
            uint32_t pos = k3 + n2 + before_i;
            if (ja) {
                const uint32_t m = m1[0] | (m1[1] << 4);
                out[pos] = (m << 8) | m | ((base + n1 + n0 - pos) << 18);
                ++pos;
            }
            if (jb) {
                const uint32_t m = m1[2] | (m1[3] << 4);
                out[pos] = (m << 8) | m | ((base + n1 + a1 + n0 + a0 - pos) << 18);
            }
            // level-3 nodes, by the first of their four lanes
            uint32_t m3 = (ja | (jb << 1)) << (2 * (lane & 3));
            m3 |= __shfl_xor_sync(FULL, m3, 1);
            m3 |= __shfl_xor_sync(FULL, m3, 2);
            if ((lane & 3) == 0 && m3) {
                const uint32_t r3 = (uint32_t)__popc(mask & ((1u << (lane >> 2)) - 1u));
                out[r3] = (m3 << 8) | m3 | ((k3 + (bi >> 23) + before_i - r3) << 18);
            }
        }
        if (vec) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int q = threadIdx.x + k * 256;
                const uint32_t m = (uint32_t)morton3((uint32_t)((q & 3) << 2), (uint32_t)((q >> 2) & 15), (uint32_t)(q >> 6));
                tile[m] = v[k].x;
                tile[m + 1] = v[k].y;
                tile[m + 8] = v[k].z;
                tile[m + 9] = v[k].w;
            }
        }
        __syncthreads();
        if (threadIdx.x < 128) {  // the four bottom-level nodes of a 32-cell word
            const uint32_t w = sb[threadIdx.x];
            uint32_t pos = node_at[threadIdx.x], child = cell_at[threadIdx.x];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t m = (w >> (8 * k)) & 0xFFu;
                if (!m) continue;
                out[pos] = (m << 8) | ((child - pos) << 18);
                ++pos;
                child += (uint32_t)__popc(m);
            }
        }
        for (int k = 0; k < 16; ++k) {
            const int c = wid * 16 + k;
            const uint32_t w = sb[c];
            if (!((w >> lane) & 1u)) continue;
            const uint32_t m = (uint32_t)(c * 32 + lane);
            uint32_t value;
            if (vec) {
                value = tile[m];
            } else {
                int x, y, z;
                brick_cell(m, x, y, z);
                value = __ldg(g.grid + (uint64_t)(gx0 + x) +
                              (uint64_t)g.w * ((uint64_t)(gy0 + y) + (uint64_t)g.h * (gz0 + z)));
            }
            out[(uint32_t)cell_at[c] + (uint32_t)__popc(w & lt)] = value;
        }
    }
}

// The same for 8^3 bricks whose voxels are already compacted (512 words a
// brick, Morton order): a warp per brick, a lane per 32-cell word of its bits.
// A brick is two waits long: its bits and its place are read together, then
// the first 128 voxels while the nodes are written.  Compacted voxel i of the
// level-2 node j goes to k + n_1(through j) + i, so the copy reads whole
// segments and needs the bounds of eight nodes only.  The 85,187 bricks of a
// mesh at 1024^3: 33 us; 47 with a read and a write of 32 cells at a time and
// the place, the bits and the voxels read one after another.
template <bool kDense>
__global__ void __launch_bounds__(256) k_place_brick8(BrickPlaces at_of, uint64_t n_dense,
                                                      const uint32_t *bits, const uint32_t *slot,
                                                      uint32_t *__restrict__ words,
                                                      uint64_t W, uint32_t *__restrict__ err) {
    chain_begin();
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const uint64_t n = kDense ? n_dense : (uint64_t)*at_of.n;
    const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t p = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < n; p += warps) {
        const uint64_t j = kDense ? p : (uint64_t)at_of.src[p];
        const uint32_t w = lane < 16 ? __ldg(bits + j * 16 + lane) : 0u;
        uint64_t b, at, size;
        brick_place<kDense>(at_of, p, b, at, size);
        const uint32_t m1 = byte_bits(w);
        const uint32_t own = (uint32_t)__popc(w) | ((uint32_t)__popc(m1) << 16);
        const uint32_t incl = warp_incl_scan(own), excl = incl - own;  // cells below, level-1 nodes above
        const uint32_t cells = __shfl_sync(FULL, incl, 31) & 0xFFFFu;
        const uint32_t *const from = slot + j * 512;
        uint32_t v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = lane + 32u * q < cells ? __ldg(from + lane + 32 * q) : 0u;
        if (size == 0) continue;
        if (at + size > W) {
            if (lane == 0) atomicOr(err, 4u);
            continue;
        }
        uint32_t *const out = words + at;
        const uint32_t other = __shfl_xor_sync(FULL, w, 1), m1o = __shfl_xor_sync(FULL, m1, 1);
        const bool first = !(lane & 1), has = (w | other) != 0u;
        const unsigned pairs = __ballot_sync(FULL, first && has);
        const uint32_t k = (uint32_t)__popc(pairs);
        // the level-2 node of this lane is its even lane and the next
        const uint32_t bj = __shfl_sync(FULL, excl, lane & ~1), tj = __shfl_sync(FULL, incl, lane | 1);
        uint32_t pos = k + (excl >> 16) + (bj & 0xFFFFu);
        uint32_t child = k + (tj >> 16) + (excl & 0xFFFFu);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const uint32_t m = (w >> (8 * t)) & 0xFFu;
            if (!m) continue;
            out[pos] = (m << 8) | ((child - pos) << 18);
            ++pos;
            child += (uint32_t)__popc(m);
        }
        if (first && has) {
            const uint32_t r = (uint32_t)__popc(pairs & lt), m = m1 | (m1o << 4);
            out[r] = (m << 8) | m | ((k + (excl >> 16) + (excl & 0xFFFFu) - r) << 18);
        }
        uint32_t through[8];  // per level-2 node: cells and level-1 nodes up to its end
#pragma unroll
        for (int q = 0; q < 8; ++q) through[q] = __shfl_sync(FULL, incl, 2 * q + 1);
        for (uint32_t i0 = 0;;) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t i = i0 + lane + 32u * q;
                uint32_t n1 = through[7] >> 16;
#pragma unroll
                for (int t = 6; t >= 0; --t)
                    if (i < (through[t] & 0xFFFFu)) n1 = through[t] >> 16;
                if (i < cells) out[k + n1 + i] = v[q];
            }
            i0 += 128;
            if (i0 >= cells) break;
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = i0 + lane + 32u * q < cells ? __ldg(from + i0 + lane + 32 * q) : 0u;
        }
    }
}

// ---- level grouping --------------------------------------------------------
//
// Every level kernel takes its element count twice: `n` from the host and
// `dn`, a device copy or nullptr.  With dn the count stays on the device
// (the small top levels are chained without host round trips); n is then an
// upper bound that sizes the arrays and the grid.

__device__ __forceinline__ uint64_t level_count(uint64_t n, const uint32_t *dn) { return dn ? (uint64_t)*dn : n; }

// head[i] = 1 where child i starts a new parent; zero for i in [count, n), so
// a scan over all n entries totals the parents.
__global__ void k_heads(const uint64_t *__restrict__ key, uint64_t n, const uint32_t *__restrict__ dn,
                        uint32_t *__restrict__ head) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t c = level_count(n, dn);
    head[i] = i < c && (i == 0 || (key[i] >> 3) != (key[i - 1] >> 3)) ? 1u : 0u;
}

__global__ void k_parents_from_heads(const uint64_t *__restrict__ ckey, uint64_t n, const uint32_t *__restrict__ dn,
                                     const uint32_t *__restrict__ head, const uint32_t *__restrict__ pidx,
                                     uint64_t *__restrict__ pkey, uint32_t *__restrict__ pstart) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= level_count(n, dn) || !head[i]) return;
    uint32_t p = pidx[i];
    pkey[p] = ckey[i] >> 3;
    pstart[p] = (uint32_t)i;
}

// pidx holds the exclusive scan of head flags: right for a head, one too high
// for the siblings after it.  Turn it into the parent index of every child.
__global__ void k_child_pidx_from_heads(const uint32_t *__restrict__ head, uint64_t n, const uint32_t *__restrict__ dn,
                                        uint32_t *__restrict__ pidx) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= level_count(n, dn)) return;
    pidx[i] = pidx[i] + head[i] - 1u;
}

// A node's subtree words and far-pointer decision (VoxelOctree.cpp:172-183)
// from its k children's subtrees; without them (bottom-level nodes) its k
// voxels.
__device__ __forceinline__ void subtree_of(uint32_t k, const uint64_t *__restrict__ childS, uint64_t *S,
                                           uint8_t *large) {
    uint64_t run = 0;
    bool far = false;
    if (childS) {
        for (uint32_t i = 0; i < k; ++i) {
            if ((uint64_t)(k - i) + run > 0x3FFFull) far = true;
            run += childS[i];
        }
    }
    *S = (uint64_t)k * (far ? 2u : 1u) + run;
    *large = far ? 1 : 0;
}

// Fused grouping of one level's children (sorted Morton keys) into parents,
// in tiles of kLvlTile children.  k_level_count counts each tile's heads
// (children whose key >> 3 differs from the previous child's); an exclusive
// scan of those counts gives each tile's first parent; k_level_emit stages
// the tile's keys in shared memory and writes every parent's key, first
// child, valid mask, child count, subtree words and far decision.  The keys are read twice and only the
// parents are written, where head flags, a scan over every child and
// separate passes for the parents, the children's parent indices and the
// masks read and wrote about three times as many bytes per child.
constexpr int kLvlThreads = 256, kLvlItems = 8, kLvlTile = kLvlThreads * kLvlItems;

__global__ void __launch_bounds__(kLvlThreads) k_level_count(const uint64_t *__restrict__ ckey, uint64_t n,
                                                             const uint32_t *__restrict__ dn,
                                                             uint32_t *__restrict__ tile_heads) {
    __shared__ uint32_t wsum[kLvlThreads / 32];
    const uint64_t c = level_count(n, dn);
    const uint64_t base = (uint64_t)blockIdx.x * kLvlTile;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint64_t k[kLvlItems], k0[kLvlItems];
    // every load issued before any is used; lane 0 also reads the child
    // before its own (the previous lane's in every other lane)
#pragma unroll
    for (int j = 0; j < kLvlItems; ++j) {
        const uint64_t i = base + (uint64_t)(j * kLvlThreads + threadIdx.x);
        k[j] = i < c ? __ldg(ckey + i) : 0ull;
        k0[j] = (lane == 0 && i > 0 && i < c) ? __ldg(ckey + i - 1) : 0ull;
    }
    uint32_t cnt = 0;
#pragma unroll
    for (int j = 0; j < kLvlItems; ++j) {
        const uint64_t i = base + (uint64_t)(j * kLvlThreads + threadIdx.x);
        uint64_t prev = __shfl_up_sync(0xffffffffu, k[j], 1);
        if (lane == 0) prev = k0[j];
        const bool head = i < c && (i == 0 || (k[j] >> 3) != (prev >> 3));
        cnt += (uint32_t)__popc(__ballot_sync(0xffffffffu, head));
    }
    if (lane == 0) wsum[wid] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
#pragma unroll
        for (int w = 0; w < kLvlThreads / 32; ++w) t += wsum[w];
        tile_heads[blockIdx.x] = t;
    }
}

// Children go through the tile in rounds of kLvlThreads, so each warp holds
// 32 consecutive children per round.  A child's parent index is the number
// of heads up to it, minus one.  A parent's run (at most 8 children) is the
// lanes from its head to the next head; three shuffle steps OR the run's
// octant bits into the head's valid mask, and the head writes the parent.
// A run that continues past its warp's 32 children ends in the next 32
// children's leading run, which that round's lane 0 has already ORed and
// counted (one table entry per round); past the tile's last round it ends
// in the keys that follow the tile, staged in shared memory.
__global__ void __launch_bounds__(kLvlThreads) k_level_emit(const uint64_t *__restrict__ ckey, uint64_t n,
                                                            const uint32_t *__restrict__ dn,
                                                            const uint32_t *__restrict__ tile_heads,
                                                            const uint32_t *__restrict__ tile_first,
                                                            const uint64_t *__restrict__ childS,
                                                            uint64_t *__restrict__ pkey, uint32_t *__restrict__ pstart,
                                                            uint8_t *__restrict__ pmask, uint8_t *__restrict__ pcount,
                                                            uint64_t *__restrict__ pS, uint8_t *__restrict__ plarge,
                                                            uint32_t *__restrict__ n_parents) {
    // sk[0]: the child before the tile; sk[1 + q]: child base + q, for q below
    // kLvlTile + 7
    __shared__ uint64_t sk[kLvlTile + 8];
    __shared__ uint32_t wpre[kLvlItems * (kLvlThreads / 32)];  // heads per (round, warp), then their exclusive prefix
    __shared__ uint16_t mh[kLvlItems][kLvlThreads];  // per child: run mask (low 8 bits) and run end lane
    __shared__ uint32_t lead[kLvlItems * (kLvlThreads / 32)];  // per round: its leading run's mask and length
    const uint64_t c = level_count(n, dn);
    const uint64_t base = (uint64_t)blockIdx.x * kLvlTile;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr int kWarps = kLvlThreads / 32;
#pragma unroll
    for (int j = 0; j < kLvlItems; ++j) {
        const int q = j * kLvlThreads + threadIdx.x;
        sk[1 + q] = base + q < c ? __ldg(ckey + base + q) : 0ull;
    }
    if (threadIdx.x < 8) {
        if (threadIdx.x == 0)
            sk[0] = (base > 0 && base - 1 < c) ? __ldg(ckey + base - 1) : 0ull;
        else {
            const uint64_t i = base + kLvlTile + threadIdx.x - 1;
            sk[kLvlTile + threadIdx.x] = i < c ? __ldg(ckey + i) : 0ull;
        }
    }
    __syncthreads();
    // heads (parent keys differ: the keys differ above their low 3 bits),
    // kept as this warp's ballot per round
    unsigned hb[kLvlItems];
#pragma unroll
    for (int j = 0; j < kLvlItems; ++j) {
        const int q = j * kLvlThreads + threadIdx.x;
        const bool head = base + q < c && (base + q == 0 || ((sk[1 + q] ^ sk[q]) & ~7ull) != 0ull);
        hb[j] = __ballot_sync(0xffffffffu, head);
        if (lane == 0) wpre[j * kWarps + wid] = (uint32_t)__popc(hb[j]);
    }
    __syncthreads();
    static_assert(kLvlItems * kWarps == 64, "one warp scans two entries per lane");
    if (wid == 0) {
        const uint32_t a0 = wpre[2 * lane], a1 = wpre[2 * lane + 1];
        uint32_t incl = a0 + a1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const uint32_t ex = incl - a0 - a1;
        wpre[2 * lane] = ex;
        wpre[2 * lane + 1] = ex + a0;
    }
    __syncthreads();
    // the tile's first parent, from a scan or by summing the earlier tiles'
    // heads here; then the last tile also leaves the level's total
    const uint32_t first = tile_first ? tile_first[blockIdx.x] : tiles_before(tile_heads, blockIdx.x);
    if (!tile_first && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
        *n_parents = first + tile_heads[blockIdx.x];
    const unsigned upto = 0xffffffffu >> (31 - lane);  // lanes 0..lane
    // Pass 2a: each lane's octant bits with its run-mates' after it, and its
    // run's end; each round's leading run (the lanes before its first head,
    // the tail of the previous round's last parent) as one table entry.
#pragma unroll
    for (int j = 0; j < kLvlItems; ++j) {
        const int q = j * kLvlThreads + threadIdx.x;
        const uint64_t i = base + q;
        const bool live = i < c;
        const uint64_t k = sk[1 + q];
        const unsigned b = hb[j];
        // a run ends at the next head or at the first lane past the last
        // child (the live lanes are a prefix of the warp's 32)
        const uint64_t w0 = base + (uint64_t)(q - lane);
        const unsigned livem = w0 >= c ? 0u : (c - w0 >= 32 ? 0xffffffffu : (1u << (uint32_t)(c - w0)) - 1u);
        const unsigned after = (b | ~livem) & ~upto;
        const int hi = after ? __ffs(after) - 1 : 32;
        // octant bits of this lane and the run-mates after it (at most 7),
        // by doubling: runs are contiguous, so lane + d in the run means the
        // lanes between are too
        unsigned m = live ? 1u << (k & 7) : 0u;
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) {
            const unsigned o = __shfl_down_sync(0xffffffffu, m, d);
            if (lane + d < hi) m |= o;
        }
        mh[j][threadIdx.x] = (uint16_t)(m | ((unsigned)hi << 8));
        if (lane == 0) lead[j * kWarps + wid] = (b & 1u) || !live ? 0u : (m | ((unsigned)hi << 8));
    }
    __syncthreads();
    // Pass 2b: the heads write their parents; a run reaching its round's last
    // lane continues in the next round's leading run (runs are at most 8
    // long), and past the tile's last round in the keys that follow it.
#pragma unroll
    for (int j = 0; j < kLvlItems; ++j) {
        const unsigned b = hb[j];
        if (!((b >> lane) & 1u)) continue;
        const int q = j * kLvlThreads + threadIdx.x;
        const uint64_t i = base + q;
        const uint64_t k = sk[1 + q];
        const unsigned v = mh[j][threadIdx.x];
        const int hi = (int)(v >> 8);
        unsigned mm = v & 0xFFu, cnt = (unsigned)(hi - lane);
        if (hi == 32) {
            const int nxt = j * kWarps + wid + 1;  // the next round of 32 children
            if (nxt < kLvlItems * kWarps) {
                const unsigned l = lead[nxt];
                mm |= l & 0xFFu;
                cnt += l >> 8;
            } else {
                for (int t = q + (int)cnt; cnt < 8 && base + t < c && ((sk[1 + t] ^ k) & ~7ull) == 0ull; ++t, ++cnt)
                    mm |= 1u << (sk[1 + t] & 7);
            }
        }
        const uint32_t p = first + wpre[j * kWarps + wid] + (uint32_t)__popc(b & upto) - 1u;
        pkey[p] = k >> 3;
        pstart[p] = (uint32_t)i;
        pmask[p] = (uint8_t)mm;
        pcount[p] = (uint8_t)cnt;
        subtree_of(cnt, childS ? childS + i : nullptr, pS + p, plarge + p);
    }
}

// Dense grouping at the cache-block level: blk_first[b] = first child of
// block b (or 0xFFFFFFFF); present = has children or top flag.
__global__ void k_block_first(const uint64_t *__restrict__ ckey, uint64_t n, const uint32_t *__restrict__ dn,
                              const uint32_t *__restrict__ head, uint32_t *__restrict__ blk_first) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= level_count(n, dn) || !head[i]) return;
    blk_first[ckey[i] >> 3] = (uint32_t)i;
}

__global__ void k_block_present(const uint32_t *__restrict__ blk_first, const uint8_t *__restrict__ topflag,
                                uint64_t nb, uint32_t *__restrict__ present) {
    uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    present[b] = (blk_first[b] != 0xFFFFFFFFu || topflag[b]) ? 1u : 0u;
}

__global__ void k_block_parents(const uint32_t *__restrict__ blk_first, const uint32_t *__restrict__ present,
                                const uint32_t *__restrict__ bidx, uint64_t nb, uint64_t n_child,
                                const uint32_t *__restrict__ dn_child, uint64_t *__restrict__ pkey,
                                uint32_t *__restrict__ pstart) {
    uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb || !present[b]) return;
    uint32_t p = bidx[b];
    pkey[p] = b;
    pstart[p] = blk_first[b] != 0xFFFFFFFFu ? blk_first[b] : (uint32_t)level_count(n_child, dn_child);
}

__global__ void k_child_pidx_from_blocks(const uint64_t *__restrict__ ckey, uint64_t n, const uint32_t *__restrict__ dn,
                                         const uint32_t *__restrict__ bidx, uint32_t *__restrict__ pidx) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= level_count(n, dn)) return;
    pidx[i] = bidx[ckey[i] >> 3];
}

// The root exists even over an empty grid: a root level with no node gets
// one, with no children (the device-count form of the host's fix-up).
__global__ void k_root_node(uint32_t *__restrict__ dn, uint64_t *__restrict__ key, uint32_t *__restrict__ start,
                            uint8_t *__restrict__ mask, uint8_t *__restrict__ count, uint64_t *__restrict__ S,
                            uint8_t *__restrict__ large) {
    if (*dn == 0) {
        *dn = 1;
        key[0] = 0;
        start[0] = 0;
        mask[0] = 0;
        count[0] = 0;
        S[0] = 0;
        large[0] = 0;
    }
}

// Per parent: valid mask and child count from its run of children.
__global__ void k_parent_masks(const uint64_t *__restrict__ pkey, const uint32_t *__restrict__ pstart, uint64_t np,
                               const uint32_t *__restrict__ dnp, const uint64_t *__restrict__ ckey, uint64_t nc,
                               const uint32_t *__restrict__ dnc, uint8_t *__restrict__ mask,
                               uint8_t *__restrict__ count) {
    uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= level_count(np, dnp)) return;
    const uint64_t c_n = level_count(nc, dnc);
    uint64_t k = pkey[p];
    uint32_t m = 0, c = 0;
    for (uint64_t i = pstart[p]; i < c_n && c < 8 && (ckey[i] >> 3) == k; ++i, ++c) m |= 1u << (ckey[i] & 7);
    mask[p] = (uint8_t)m;
    count[p] = (uint8_t)c;
}

// The same per parent from its children, one thread per child: the lanes
// holding one parent's children (a run, at most 8) find each other with a
// match and OR their octant bits into the parent's valid mask with one warp
// reduction.  The run's first lane writes mask and count; a run that started
// in the previous warp is that warp's to write, and one that continues past
// this warp is finished by reading its remaining children (at most 7).
// Parents without children (cache blocks only the top table marks, an empty
// root) are zeroed beforehand.
__global__ void k_parent_masks_warp(const uint64_t *__restrict__ ckey, uint64_t nc, const uint32_t *__restrict__ dnc,
                                    const uint32_t *__restrict__ pidx, uint8_t *__restrict__ mask,
                                    uint8_t *__restrict__ count) {
    const uint64_t n = level_count(nc, dnc);
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned lane = threadIdx.x & 31u;
    const bool live = i < n;
    const uint32_t p = live ? pidx[i] : 0xFFFFFFFFu;
    const unsigned peers = __match_any_sync(0xffffffffu, p);
    const unsigned m = __reduce_or_sync(peers, live ? 1u << (ckey[i] & 7) : 0u);
    if (!live || lane != (unsigned)(__ffs(peers) - 1)) return;
    if (lane == 0 && i > 0 && pidx[i - 1] == p) return;
    unsigned mm = m, c = (unsigned)__popc(peers);
    for (uint64_t k = i + c; k < n && c < 8 && pidx[k] == p; ++k, ++c) mm |= 1u << (ckey[k] & 7);
    mask[p] = (uint8_t)mm;
    count[p] = (uint8_t)c;
}

// ---- subtree sizes and far-pointer decisions (bottom-up) -------------------

__global__ void k_subtree(uint64_t np, const uint32_t *__restrict__ dnp, const uint8_t *__restrict__ count,
                          const uint32_t *__restrict__ pstart, const uint64_t *__restrict__ childS, int bottom,
                          uint64_t *__restrict__ S, uint8_t *__restrict__ large) {
    uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= level_count(np, dnp)) return;
    subtree_of(count[p], bottom ? nullptr : childS + pstart[p], S + p, large + p);
}

// ---- placement (top-down) ---------------------------------------------------

__global__ void k_root_word(const uint8_t *__restrict__ mask, const uint8_t *__restrict__ large, int root_is_bottom,
                            uint64_t *__restrict__ B, uint32_t *__restrict__ words) {
    B[0] = 1;
    uint32_t m = mask[0];
    words[0] = (m << 8) | (root_is_bottom ? 0u : m) | (large[0] ? 0x10000u : 0u) | (1u << 18);
}

// Parents at one level place their (internal) children and write the
// children's descriptors; child_is_bottom selects leafMask = 0.
// Every word write is checked against W; a violation (an internal
// inconsistency) is skipped and reported through *err.
__global__ void k_place(uint64_t np, const uint32_t *__restrict__ dnp, const uint8_t *__restrict__ count,
                        const uint32_t *__restrict__ pstart, const uint8_t *__restrict__ plarge,
                        const uint64_t *__restrict__ pB, const uint64_t *__restrict__ cS,
                        const uint8_t *__restrict__ cmask, const uint8_t *__restrict__ clarge, int child_is_bottom,
                        uint64_t *__restrict__ cB, uint32_t *__restrict__ words, uint64_t W,
                        uint32_t *__restrict__ err) {
    uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= level_count(np, dnp)) return;
    uint32_t k = count[p];
    bool far = plarge[p] != 0;
    uint64_t stride = far ? 2 : 1;
    uint64_t B = pB[p];
    uint64_t run = 0;
    uint32_t s0 = pstart[p];
    for (uint32_t i = 0; i < k; ++i) {
        uint32_t c = s0 + i;
        uint64_t pos = B + (uint64_t)i * stride;
        uint64_t blk = B + (uint64_t)k * stride + run;
        run += cS[c];
        cB[c] = blk;
        uint64_t off = blk - pos;
        uint32_t m = cmask[c];
        uint32_t w = (m << 8) | (child_is_bottom ? 0u : m) | (clarge[c] ? 0x10000u : 0u);
        if (pos + (far ? 1 : 0) >= W) {
            atomicOr(err, 1u);
            continue;
        }
        if (far) {
            w |= 0x20000u | (uint32_t)((off >> 32) << 18);
            words[pos + 1] = (uint32_t)off;
        } else {
            w |= (uint32_t)(off << 18);
        }
        words[pos] = w;
    }
}

__global__ void k_place_leaves(uint64_t n, const uint32_t *__restrict__ pidx, uint64_t np,
                               const uint32_t *__restrict__ dnp, const uint32_t *__restrict__ pstart,
                               const uint64_t *__restrict__ pB, const uint32_t *__restrict__ payload,
                               uint32_t *__restrict__ words, uint64_t W, uint32_t *__restrict__ err) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t p = pidx[i];
    if (p >= level_count(np, dnp) || i < pstart[p] || i - pstart[p] >= 8) {
        atomicOr(err, 2u);
        return;
    }
    uint64_t dst = pB[p] + (i - pstart[p]);
    if (dst >= W) {
        atomicOr(err, 4u);
        return;
    }
    words[dst] = payload[i];
}

// The same placement with a lane per child: a warp takes per_warp consecutive
// parents (32, or 4 where a level has too few to fill the chip: their
// children then fit one round of the serial loop below), whose children follow one another (at most 256), marks which lane
// owns each child in a per-warp table, and places the children 32 at a time.
// A child's block offset is the sum of the subtree sizes of its earlier
// siblings: a segmented scan over the round's lanes (runs are at most 8
// long, so three shuffle steps), plus what a run that began in the previous
// round carried over.  The descriptors and far words are those of k_place.
__global__ void __launch_bounds__(256) k_place_warp(uint64_t np, const uint32_t *__restrict__ dnp,
                                                    const uint8_t *__restrict__ count,
                                                    const uint32_t *__restrict__ pstart,
                                                    const uint8_t *__restrict__ plarge,
                                                    const uint64_t *__restrict__ pB, const uint64_t *__restrict__ cS,
                                                    const uint8_t *__restrict__ cmask,
                                                    const uint8_t *__restrict__ clarge, int child_is_bottom,
                                                    uint64_t nc, const uint32_t *__restrict__ dnc, int per_warp,
                                                    uint64_t *__restrict__ cB, uint32_t *__restrict__ words,
                                                    uint64_t W, uint32_t *__restrict__ err) {
    __shared__ uint8_t owner[8][256];  // per warp: the lane whose parent holds child s0 + i
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned upto = 0xffffffffu >> (31 - lane);
    const uint64_t n = level_count(np, dnp);
    const uint64_t p0 = ((uint64_t)blockIdx.x * 8 + wid) * per_warp;
    if (p0 >= n) return;  // uniform per warp
    const uint64_t p = p0 + lane;
    const bool live = lane < per_warp && p < n;
    const uint32_t k = live ? count[p] : 0u;
    const uint32_t stride = (live && plarge[p]) ? 2u : 1u;
    const uint64_t s = live ? pstart[p] : 0ull, B = live ? pB[p] : 0ull;
    // parents without children (cache blocks only the top table marks) have
    // none to place; the others' children follow one another
    const unsigned runs = __ballot_sync(0xffffffffu, k != 0);
    if (!runs) return;
    const uint64_t s0 = __shfl_sync(0xffffffffu, s, __ffs(runs) - 1);
    uint32_t before = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += t;
    }
    before -= k;
    const bool bad = k != 0 && (s != s0 + before || s + k > level_count(nc, dnc));
    if (__any_sync(0xffffffffu, bad)) {
        if (bad) atomicOr(err, 2u);
        return;
    }
    for (uint32_t j = 0; j < k; ++j) owner[wid][before + j] = (uint8_t)lane;
    const uint32_t total = __reduce_max_sync(0xffffffffu, k ? before + k : 0u);
    __syncwarp();
    uint64_t carry = 0;  // subtree sizes of the earlier siblings of the round's first child, from earlier rounds
    for (uint32_t i0 = 0; i0 < total; i0 += 32) {
        const uint32_t i = i0 + lane;
        const bool in = i < total;
        const int l = in ? owner[wid][i] : 0;
        const uint64_t c = s0 + i;
        const uint64_t S = in ? cS[c] : 0ull;
        // the lanes of one parent in this round form a segment
        const bool start = !in || lane == 0 || owner[wid][i - 1] != (uint8_t)l;
        const unsigned starts = __ballot_sync(0xffffffffu, start);
        const int lo = 31 - __clz((int)(starts & upto));
        uint64_t incl = S;
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) {
            const uint64_t t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane - d >= lo) incl += t;
        }
        const uint64_t Bl = __shfl_sync(0xffffffffu, B, l);
        const uint64_t sl = __shfl_sync(0xffffffffu, s, l);
        const uint32_t kl = __shfl_sync(0xffffffffu, k, l);
        const uint32_t stl = __shfl_sync(0xffffffffu, stride, l);
        // the first segment continues a run from the previous round when its
        // first child is not its parent's first
        const uint64_t add = (lo == 0 && i0 > 0 && s0 + i0 != sl) ? carry : 0ull;
        const uint64_t run = add + incl - S;
        // what the last lane's run carries into the next round
        const uint64_t last_total = __shfl_sync(0xffffffffu, add + incl, 31);
        carry = last_total;
        if (in) {
            const uint64_t jj = c - sl;
            const uint64_t pos = Bl + jj * stl;
            const uint64_t blk = Bl + (uint64_t)kl * stl + run;
            cB[c] = blk;
            const uint64_t off = blk - pos;
            const uint32_t m = cmask[c];
            uint32_t w = (m << 8) | (child_is_bottom ? 0u : m) | (clarge && clarge[c] ? 0x10000u : 0u);
            if (pos + (stl == 2u ? 1u : 0u) >= W) {
                atomicOr(err, 1u);
            } else {
                if (stl == 2u) {
                    w |= 0x20000u | (uint32_t)((off >> 32) << 18);
                    words[pos + 1] = (uint32_t)off;
                } else {
                    w |= (uint32_t)(off << 18);
                }
                words[pos] = w;
            }
        }
    }
}

// The leaves: every bottom-level parent's run of leaf words goes into its
// child block, in key order (the slots k_place_leaves fills one leaf at a
// time).  A warp takes 32 consecutive parents, whose runs are consecutive
// (each starts where the previous one ends), so their at most 256 leaves are
// one range: each lane marks its run's slots in a per-warp owner table, then
// the warp copies the range with consecutive lanes on consecutive leaves.
// A run reaching past the word count or the leaves is reported through *err.
__global__ void __launch_bounds__(256) k_place_leaf_runs(uint64_t np, const uint32_t *__restrict__ dnp,
                                                         const uint8_t *__restrict__ count,
                                                         const uint32_t *__restrict__ pstart,
                                                         const uint64_t *__restrict__ pB,
                                                         const uint32_t *__restrict__ payload, uint64_t n_leaves,
                                                         uint32_t *__restrict__ words, uint64_t W,
                                                         uint32_t *__restrict__ err) {
    __shared__ uint8_t owner[8][256];  // per warp: the lane whose parent holds leaf slot s0 + i
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint64_t n = level_count(np, dnp);
    const uint64_t p0 = ((uint64_t)blockIdx.x * blockDim.x) + (uint64_t)wid * 32;
    if (p0 >= n) return;  // uniform per warp
    const uint64_t p = p0 + lane;
    const bool live = p < n;
    const uint32_t k = live ? count[p] : 0u;
    const uint64_t s = live ? pstart[p] : 0ull, B = live ? pB[p] : 0ull;
    // parents without children (cache blocks only the top table marks) have
    // no run; the others' runs follow one another from the first one's start
    const unsigned runs = __ballot_sync(0xffffffffu, k != 0);
    if (!runs) return;
    const uint64_t s0 = __shfl_sync(0xffffffffu, s, __ffs(runs) - 1);
    // the runs must tile the range in lane order: each starts where the
    // earlier lanes' runs end
    uint32_t before = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += t;
    }
    before -= k;
    const bool bad = k != 0 && (B + k > W || s + k > n_leaves || s != s0 + before);
    if (__any_sync(0xffffffffu, bad)) {
        if (bad) atomicOr(err, 4u);
        return;
    }
    const uint32_t rel = k ? (uint32_t)(s - s0) : 0u;
    for (uint32_t j = 0; j < k; ++j) owner[wid][rel + j] = (uint8_t)lane;
    const uint32_t total = __reduce_max_sync(0xffffffffu, k ? rel + k : 0u);
    __syncwarp();
    // every lane takes the same number of rounds: the shuffles read lanes
    // that may own no leaf of the round
    for (uint32_t i0 = 0; i0 < total; i0 += 32) {
        const uint32_t i = i0 + lane;
        const int l = i < total ? owner[wid][i] : 0;
        const uint64_t Bl = __shfl_sync(0xffffffffu, B, l);
        const uint64_t sl = __shfl_sync(0xffffffffu, s, l);
        if (i < total) words[Bl + (s0 + i - sl)] = payload[s0 + i];
    }
}

// ---- dense pyramid over bricks ------------------------------------------------
//
// Above bricks the levels hold few nodes: a 2048^3 cube has 2 M bricks and
// 300,000 nodes above them.  Up to kPyramidBits bits of brick code, every
// level is an array over all its cells in Morton order (8 consecutive cells
// are one parent's children), which needs no keys, no scans and no grouping:
// one thread per parent going up, one per child coming down.  Levels of at
// most kTopCells children are handled by one CTA in one launch: with so few
// nodes a level is its launch and one round of memory latency.
//
// A 512^3 sphere union of 37 M voxels (42.6 M words) took 55 launches and 544
// us of kernels through voxel keys, sorted levels and node arrays, and takes
// 6 launches and 172 us through bricks: 87 for the bits, 59 to place the
// bricks, 26 for the five levels above.  Beyond kPyramidBits (a 4096^3 cube or
// a thin grid in one) the arrays would grow with the cube and not with what it
// holds, so the bricks are compacted and go through the sorted levels.  The
// line lies at the largest cubes measured (2048^3 grids, 1024^3 meshes, whose
// table of brick counts it bounds too); a cube just past it has not been timed
// in this form.
constexpr int kPyramidBits = 21;
constexpr uint32_t kTopCells = 4096, kTopPlaced = 512;  // going up, coming down
constexpr int kPyramidMax = kPyramidBits / 3 + 1;  // levels, bricks included

struct Pyramid {
    int base, top;             // level of the bricks, of the root
    const uint32_t *words_of;  // bricks: subtree words ...
    const uint8_t *mask_of;    // ... node mask ...
    const uint8_t *any_of;     // ... and presence (null: a brick with words)
    uint64_t *S[kPyramidMax];  // level base + l: subtree words (l >= 1)
    uint64_t *B[kPyramidMax];  // child block position
    uint8_t *mask[kPyramidMax], *meta[kPyramidMax];  // valid mask; bit 0 present, bit 1 its children are far
    const uint8_t *topflag;    // cache blocks that exist at level log_block, or null
    int log_block;
};

__device__ __forceinline__ uint32_t pyramid_cells(const Pyramid &p, int level) { return 1u << (3 * (p.top - level)); }

// Node `c` of `level` from its children (VoxelOctree.cpp:139-183).
__device__ __forceinline__ void pyramid_node(const Pyramid &p, int level, uint32_t c) {
    const int l = level - p.base;
    uint32_t mask = 0;
    uint64_t s[8];
    if (l == 1) {
        const uint4 a = reinterpret_cast<const uint4 *>(p.words_of)[2 * c], b = reinterpret_cast<const uint4 *>(p.words_of)[2 * c + 1];
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint2 any = make_uint2(0u, 0u);
        if (p.any_of) any = reinterpret_cast<const uint2 *>(p.any_of)[c];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            s[i] = w[i];
            const uint32_t there = p.any_of ? ((i < 4 ? any.x : any.y) >> (8 * (i & 3))) & 255u : w[i];
            mask |= there ? 1u << i : 0u;
        }
    } else {
        const uint2 m = reinterpret_cast<const uint2 *>(p.meta[l - 1])[c];
        const ulonglong2 *q = reinterpret_cast<const ulonglong2 *>(p.S[l - 1] + 8ull * c);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const ulonglong2 v = q[i];
            s[2 * i] = v.x;
            s[2 * i + 1] = v.y;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) mask |= (((i < 4 ? m.x : m.y) >> (8 * (i & 3))) & 1u) << i;
    }
    const uint32_t k = (uint32_t)__popc(mask);
    uint64_t run = 0;
    uint32_t r = 0;
    bool far = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (!((mask >> i) & 1u)) continue;
        if ((uint64_t)(k - r) + run > 0x3FFFull) far = true;
        run += s[i];
        ++r;
    }
    const bool present = mask != 0 || level == p.top || (p.topflag && level == p.log_block && p.topflag[c] != 0);
    p.mask[l][c] = (uint8_t)mask;
    p.meta[l][c] = (uint8_t)((present ? 1u : 0u) | (far ? 2u : 0u));
    p.S[l][c] = (uint64_t)k * (far ? 2u : 1u) + run;
}

// Cell `c` of `level` (whole warps call, the 8 lanes of a parent together;
// cells past the level's do nothing): its position in its parent's child
// block, its descriptor there and its own child block's position
// (VoxelOctree.cpp:184-205).
__device__ __forceinline__ void pyramid_place(const Pyramid &p, int level, uint32_t c, uint32_t *__restrict__ words,
                                              uint64_t W, uint32_t *__restrict__ err) {
    const int l = level - p.base;
    const bool in = c < pyramid_cells(p, level);
    const uint32_t i = c & 7u, up = in ? c >> 3 : 0u;
    const uint32_t mask = in ? p.mask[l + 1][up] : 0u, meta = p.meta[l + 1][up];
    const uint64_t B = p.B[l + 1][up];
    const bool there = (mask >> i) & 1u;
    const uint64_t S = !there ? 0ull : (l == 0 ? (uint64_t)p.words_of[c] : p.S[l][c]);
    uint64_t incl = S;
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) {
        const uint64_t t = __shfl_up_sync(0xffffffffu, incl, d, 8);
        if (i >= (uint32_t)d) incl += t;
    }
    if (!there) return;
    const uint32_t k = (uint32_t)__popc(mask), r = (uint32_t)__popc(mask & ((1u << i) - 1u)), stride = (meta & 2u) ? 2u : 1u;
    const uint64_t pos = B + (uint64_t)r * stride, blk = B + (uint64_t)k * stride + (incl - S), off = blk - pos;
    p.B[l][c] = blk;
    const uint32_t m = l == 0 ? p.mask_of[c] : p.mask[l][c];
    uint32_t w = (m << 8) | m | (l > 0 && (p.meta[l][c] & 2u) ? 0x10000u : 0u);
    if (pos + stride > W) {
        atomicOr(err, 1u);
        return;
    }
    if (stride == 2u) {
        w |= 0x20000u | (uint32_t)((off >> 32) << 18);
        words[pos + 1] = (uint32_t)off;
    } else {
        w |= (uint32_t)(off << 18);
    }
    words[pos] = w;
}

__global__ void __launch_bounds__(256) k_pyramid_up(Pyramid p, int level) {
    chain_begin();
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < pyramid_cells(p, level)) pyramid_node(p, level, c);
}

// The levels from `level` up to the root.  Reports the root's subtree words
// and, where counted, the voxels.
__global__ void __launch_bounds__(512) k_pyramid_top_up(Pyramid p, int level, const unsigned long long *n_voxels,
                                                        uint64_t *report) {
    chain_begin();
    for (; level <= p.top; ++level) {
        for (uint32_t c = threadIdx.x; c < pyramid_cells(p, level); c += blockDim.x) pyramid_node(p, level, c);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        report[0] = p.S[p.top - p.base][0];
        report[1] = n_voxels ? *n_voxels : 0;
    }
}

__global__ void __launch_bounds__(256) k_pyramid_down(Pyramid p, int level, uint32_t *__restrict__ words, uint64_t W,
                                                      uint32_t *__restrict__ err) {
    chain_begin();
    pyramid_place(p, level, blockIdx.x * blockDim.x + threadIdx.x, words, W, err);
}

// The root and every level down to `level`.
__global__ void __launch_bounds__(kTopPlaced) k_pyramid_top_down(Pyramid p, int level, uint32_t *__restrict__ words,
                                                           uint64_t W, uint32_t *__restrict__ err) {
    const int t = p.top - p.base;
    if (threadIdx.x == 0) {
        const uint32_t m = t ? p.mask[t][0] : p.mask_of[0];
        words[0] = (m << 8) | m | (t && (p.meta[t][0] & 2u) ? 0x10000u : 0u) | (1u << 18);
        p.B[t][0] = 1;
    }
    __syncthreads();
    for (int e = p.top - 1; e >= level; --e) {
        for (uint32_t c0 = 0; c0 < pyramid_cells(p, e); c0 += blockDim.x) pyramid_place(p, e, c0 + threadIdx.x, words, W, err);
        __syncthreads();
    }
}

inline unsigned blocks_for(uint64_t n, int t = 256) {
    uint64_t b = (n + t - 1) / t;
    return (unsigned)(b ? b : 1);  // kernels check their own bounds; never launch an empty grid
}

#define SVO_LAUNCH_CHECK(name)                                        \
    do {                                                              \
        cudaError_t _e = cudaGetLastError();                          \
        if (_e != cudaSuccess) return ::svo::cuda_fail(_e, "launch of " name); \
    } while (0)

// Bump allocator over a few pool chunks for the level build's many
// short-lived arrays.  One stream-ordered allocation and free per array cost
// about 240 driver calls per build, most of them right after a host
// synchronisation, when the GPU waits on the host.  The chunks return to the
// pool (stream-ordered) when the arena is destroyed, after every launch that
// uses them has been enqueued.
class BuildArena {
public:
    explicit BuildArena(cudaStream_t s) : st_(s) {}
    BuildArena(const BuildArena &) = delete;
    BuildArena &operator=(const BuildArena &) = delete;
    ~BuildArena() {
        for (void *c : chunks_) cudaFreeAsync(c, st_);
    }
    cudaError_t alloc(void **p, size_t bytes) {
        bytes = (bytes + 255) & ~size_t(255);
        if (bytes > left_) {
            const size_t cb = std::max(bytes, kChunk);
            void *c = nullptr;
            cudaError_t e = scratch_alloc(&c, cb, st_);
            if (e != cudaSuccess) return e;
            chunks_.push_back(c);
            cur_ = static_cast<char *>(c);
            left_ = cb;
        }
        *p = cur_;
        cur_ += bytes;
        left_ -= bytes;
        return cudaSuccess;
    }

private:
    static constexpr size_t kChunk = size_t(64) << 20;
    cudaStream_t st_;
    std::vector<void *> chunks_;
    char *cur_ = nullptr;
    size_t left_ = 0;
};

// Stream-ordered temporary buffer, from the pool or from a BuildArena.
template <typename T>
struct DevBuf {
    T *p = nullptr;
    cudaStream_t st = nullptr;
    bool owned = false;  // false: memory of a BuildArena (freed with the arena)
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    cudaError_t alloc(uint64_t n, cudaStream_t s) {
        st = s;
        owned = true;
        return scratch_alloc((void **)&p, (size_t)(n ? n : 1) * sizeof(T), s);
    }
    cudaError_t alloc(uint64_t n, BuildArena &a) {
        owned = false;
        return a.alloc((void **)&p, (size_t)(n ? n : 1) * sizeof(T));
    }
    void release() {
        if (p && owned) cudaFreeAsync(p, st);
        p = nullptr;
    }
    ~DevBuf() { release(); }
};

struct LevelArrays {
    uint64_t n = 0;                // node count, or its upper bound when dn != nullptr
    const uint32_t *dn = nullptr;  // the node count on the device (levels chained without round trips)
    DevBuf<uint64_t> key;
    DevBuf<uint32_t> start;
    DevBuf<uint8_t> mask, count, large;
    DevBuf<uint64_t> S, B;  // subtree words; child block position (placement)
    cudaError_t alloc(uint64_t nodes, BuildArena &a) {
        cudaError_t e = key.alloc(nodes, a);
        if (e == cudaSuccess) e = start.alloc(nodes, a);
        if (e == cudaSuccess) e = mask.alloc(nodes, a);
        if (e == cudaSuccess) e = count.alloc(nodes, a);
        if (e == cudaSuccess) e = large.alloc(nodes, a);
        if (e == cudaSuccess) e = S.alloc(nodes, a);
        return e;
    }
};

#define SVO_TRY_ALLOC(expr)                                                   \
    do {                                                                      \
        cudaError_t _e = (expr);                                              \
        if (_e != cudaSuccess) return ::svo::cuda_fail(_e, "device allocation in build"); \
    } while (0)

template <typename TO>
int scan_to(const uint32_t *in, TO *out, uint64_t n, TO *total_host, cudaStream_t st, BuildArena *arena = nullptr) {
    DevBuf<TO> scratch, tot;
    if (arena) {
        SVO_TRY_ALLOC(scratch.alloc(scan_scratch_elems(n), *arena));
        SVO_TRY_ALLOC(tot.alloc(1, *arena));
    } else {
        SVO_TRY_ALLOC(scratch.alloc(scan_scratch_elems(n), st));
        SVO_TRY_ALLOC(tot.alloc(1, st));
    }
    SVO_CUDA_TRY((exclusive_scan<uint32_t, TO>(in, out, n, tot.p, scratch.p, st)));
    SVO_CUDA_TRY(cudaMemcpyAsync(total_host, tot.p, sizeof(TO), cudaMemcpyDeviceToHost, st));
    SVO_CUDA_TRY(cudaStreamSynchronize(st));
    return SVO_OK;
}

// Exclusive scan with the total left on the device (no round trip).
template <typename TO>
int scan_on_device(const uint32_t *in, TO *out, uint64_t n, TO *d_total, cudaStream_t st, BuildArena &arena) {
    DevBuf<TO> scratch;
    SVO_TRY_ALLOC(scratch.alloc(scan_scratch_elems(n), arena));
    SVO_CUDA_TRY((exclusive_scan<uint32_t, TO>(in, out, n, d_total, scratch.p, st)));
    return SVO_OK;
}

// Levels whose children number at most this many are chained on the device.
constexpr uint64_t kDeviceLevels = 1ull << 20;

// Parents per warp of k_place_warp: 4 while that many warps fit the chip at
// once (152 SMs x 64), else 32.
int parents_per_warp(uint64_t n) { return n <= 4ull * 152 * 64 ? 4 : 32; }

// Phases 2 and 3 above level `base` (see the top): the levels base + 1 .. D grouped
// bottom-up with their subtree sizes, then the words allocated, the levels
// placed top-down, and place_base(words, W, err) writes what lies below the
// base nodes' descriptors.  Level 0 is the voxels (leaf_keys, n_leaves);
// above it lv[base] comes with key, mask, count and S (large: none), and its
// count on the device (dn).  n_voxels: optionally, the voxels' total on the
// device, refused at 2^32-1 and more.
template <typename PlaceBase>
int build_levels(std::vector<LevelArrays> &lv, int base, const uint64_t *leaf_keys, uint64_t n_leaves, int D,
                 int log_block, const uint8_t *d_topflag, BuildArena &arena, cudaStream_t st,
                 const unsigned long long *n_voxels, PlaceBase place_base, uint32_t **d_words_out,
                 uint64_t *n_words_out) {
    const bool multi_block = log_block < D;
    const uint64_t n_blocks = multi_block ? (1ull << (3 * (D - log_block))) : 0;
    if (multi_block && !d_topflag) return set_error(SVO_ERR_INVALID, "build: missing cache-block flags");
    int rc = SVO_OK;

    // While a level's children number more than kDeviceLevels, the parent
    // count is read back (exact array sizes).  From the first level with
    // fewer children on, and everywhere above bricks, the counts stay on the
    // device (dcount[e]) and the arrays are sized by upper bounds: no host
    // round trip per level.
    DevBuf<uint32_t> dcount;
    SVO_TRY_ALLOC(dcount.alloc(D + 1, arena));
    const uint64_t *ckey = base ? lv[base].key.p : leaf_keys;
    uint64_t nc = base ? lv[base].n : n_leaves;  // children: exact count, or an upper bound when cdn != nullptr
    const uint32_t *cdn = base ? lv[base].dn : nullptr;  // device count of the children
    bool on_device = cdn != nullptr;
    for (int e = base + 1; e <= D; ++e) {
        LevelArrays &L = lv[e];
        const uint64_t *childS = e > 1 ? lv[e - 1].S.p : nullptr;
        if (!on_device && nc <= kDeviceLevels) on_device = true;
        uint32_t *dn = on_device ? dcount.p + e : nullptr;
        // at most one node per cell of edge 2^e, and never more parents than children
        const uint64_t cells = 3 * (D - e) >= 63 ? ~0ull : 1ull << (3 * (D - e));
        if (multi_block && e == log_block) {
            // Dense grouping over cache blocks, adding blocks that only the top
            // lookup table marks (descriptors without children).
            DevBuf<uint32_t> head, pidx, first, present, bidx;
            SVO_TRY_ALLOC(head.alloc(nc, arena));
            SVO_TRY_ALLOC(pidx.alloc(nc, arena));
            SVO_TRY_ALLOC(first.alloc(n_blocks, arena));
            SVO_TRY_ALLOC(present.alloc(n_blocks, arena));
            SVO_TRY_ALLOC(bidx.alloc(n_blocks, arena));
            if (nc) {
                k_heads<<<blocks_for(nc), 256, 0, st>>>(ckey, nc, cdn, head.p);
                SVO_LAUNCH_CHECK("k_heads");
            }
            SVO_CUDA_TRY(cudaMemsetAsync(first.p, 0xFF, n_blocks * sizeof(uint32_t), st));
            if (nc) k_block_first<<<blocks_for(nc), 256, 0, st>>>(ckey, nc, cdn, head.p, first.p);
            k_block_present<<<blocks_for(n_blocks), 256, 0, st>>>(first.p, d_topflag, n_blocks, present.p);
            SVO_LAUNCH_CHECK("k_block_present");
            if (on_device) {
                rc = scan_on_device<uint32_t>(present.p, bidx.p, n_blocks, dn, st, arena);
                L.n = n_blocks;
            } else {
                uint32_t np = 0;
                rc = scan_to<uint32_t>(present.p, bidx.p, n_blocks, &np, st, &arena);
                L.n = np;
            }
            if (rc) return rc;
            if (e == D && L.n == 0) L.n = 1;  // the root (fixed up below)
            SVO_TRY_ALLOC(L.alloc(L.n, arena));
            // blocks only the top table marks keep mask and count 0
            SVO_CUDA_TRY(cudaMemsetAsync(L.mask.p, 0, L.n, st));
            SVO_CUDA_TRY(cudaMemsetAsync(L.count.p, 0, L.n, st));
            k_block_parents<<<blocks_for(n_blocks), 256, 0, st>>>(first.p, present.p, bidx.p, n_blocks, nc, cdn,
                                                                  L.key.p, L.start.p);
            if (nc) {
                k_child_pidx_from_blocks<<<blocks_for(nc), 256, 0, st>>>(ckey, nc, cdn, bidx.p, pidx.p);
                k_parent_masks_warp<<<blocks_for(nc), 256, 0, st>>>(ckey, nc, cdn, pidx.p, L.mask.p, L.count.p);
                SVO_LAUNCH_CHECK("k_parent_masks_warp");
            }
            k_subtree<<<blocks_for(L.n), 256, 0, st>>>(L.n, dn, L.count.p, L.start.p, childS, e == 1, L.S.p, L.large.p);
            SVO_LAUNCH_CHECK("k_subtree");
        } else {
            // Fused grouping: tile head counts, their scan (a few tiles sum
            // the earlier ones themselves), then the parents.
            const uint64_t tiles = (nc + kLvlTile - 1) / kLvlTile;
            const bool self = on_device && tiles <= kSelfScanTiles;
            DevBuf<uint32_t> th, tf;
            SVO_TRY_ALLOC(th.alloc(tiles, arena));
            if (!self) SVO_TRY_ALLOC(tf.alloc(tiles, arena));
            if (nc) {
                k_level_count<<<(unsigned)tiles, kLvlThreads, 0, st>>>(ckey, nc, cdn, th.p);
                SVO_LAUNCH_CHECK("k_level_count");
            }
            if (on_device) {
                if (!tiles)
                    SVO_CUDA_TRY(cudaMemsetAsync(dn, 0, sizeof(uint32_t), st));
                else if (!self)
                    rc = scan_on_device<uint32_t>(th.p, tf.p, tiles, dn, st, arena);
                L.n = std::min(nc, cells);
            } else {
                uint32_t np = 0;
                if (tiles) rc = scan_to<uint32_t>(th.p, tf.p, tiles, &np, st, &arena);
                L.n = np;
            }
            if (rc) return rc;
            if (e == D && L.n == 0) L.n = 1;  // the root (fixed up below)
            SVO_TRY_ALLOC(L.alloc(L.n, arena));
            if (nc) {
                k_level_emit<<<(unsigned)tiles, kLvlThreads, 0, st>>>(ckey, nc, cdn, th.p, self ? nullptr : tf.p, childS,
                                                                    L.key.p, L.start.p, L.mask.p, L.count.p, L.S.p,
                                                                    L.large.p, dn);
                SVO_LAUNCH_CHECK("k_level_emit");
            }
        }
        L.dn = dn;
        ckey = L.key.p;
        nc = L.n;
        cdn = L.dn;
    }
    // The root always exists, even over an empty grid (its level's count is
    // on the device: it has at most 8 children).
    k_root_node<<<1, 1, 0, st>>>(const_cast<uint32_t *>(lv[D].dn), lv[D].key.p, lv[D].start.p, lv[D].mask.p,
                                 lv[D].count.p, lv[D].S.p, lv[D].large.p);
    SVO_LAUNCH_CHECK("k_root_node");

    uint64_t S_root = 0;
    unsigned long long voxels = 0;
    SVO_CUDA_TRY(cudaMemcpyAsync(&S_root, lv[D].S.p, sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    if (n_voxels) SVO_CUDA_TRY(cudaMemcpyAsync(&voxels, n_voxels, sizeof(voxels), cudaMemcpyDeviceToHost, st));
    SVO_CUDA_TRY(cudaStreamSynchronize(st));
    if (voxels >= 0xFFFFFFFFull) return set_error(SVO_ERR_LIMIT, "%llu occupied voxels exceed 2^32-1", voxels);
    const uint64_t W = 1 + S_root;

    uint32_t *words = nullptr;
    SVO_CUDA_TRY(alloc_words(&words, W, st));
    auto place = [&]() -> int {
        DevBuf<uint32_t> err;
        SVO_TRY_ALLOC(err.alloc(1, arena));
        SVO_CUDA_TRY(cudaMemsetAsync(err.p, 0, sizeof(uint32_t), st));
        SVO_TRY_ALLOC(lv[D].B.alloc(1, arena));
        k_root_word<<<1, 1, 0, st>>>(lv[D].mask.p, lv[D].large.p, D == 1, lv[D].B.p, words);
        SVO_LAUNCH_CHECK("k_root_word");
        for (int e = D; e > std::max(base, 1); --e) {
            LevelArrays &P = lv[e];
            LevelArrays &C = lv[e - 1];
            SVO_TRY_ALLOC(C.B.alloc(C.n, arena));
            const int ppw = parents_per_warp(P.n);
            k_place_warp<<<blocks_for(P.n, 8 * ppw), 256, 0, st>>>(P.n, P.dn, P.count.p, P.start.p, P.large.p, P.B.p,
                                                                  C.S.p, C.mask.p, C.large.p, e - 1 == 1, C.n, C.dn,
                                                                  ppw, C.B.p, words, W, err.p);
            SVO_LAUNCH_CHECK("k_place_warp");
        }
        int r = place_base(words, W, err.p);
        if (r) return r;
        uint32_t err_h = 0;
        SVO_CUDA_TRY(cudaMemcpyAsync(&err_h, err.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        SVO_CUDA_TRY(cudaStreamSynchronize(st));
        if (err_h) return set_error(SVO_ERR_DEVICE, "octree build placement check failed (flags %u)", err_h);
        return SVO_OK;
    };
    rc = place();
    if (rc) {
        free_words(words, W, st);
        return rc;
    }
    *d_words_out = words;
    *n_words_out = W;
    return SVO_OK;
}

// The kept bricks (at most `most` of them) as nodes of their level, with the
// count on the device, and their own indices in `src`.
int keep_bricks(const BrickNodes &b, uint64_t most, LevelArrays &L, DevBuf<uint32_t> &src, DevBuf<uint32_t> &n_kept,
                BuildArena &arena, cudaStream_t st) {
    const uint64_t tiles = (b.n + kNodeTile - 1) / kNodeTile;
    L.n = std::max<uint64_t>(most, 1);
    SVO_TRY_ALLOC(n_kept.alloc(1, arena));
    SVO_TRY_ALLOC(src.alloc(L.n, arena));
    SVO_TRY_ALLOC(L.key.alloc(L.n, arena));
    SVO_TRY_ALLOC(L.mask.alloc(L.n, arena));
    SVO_TRY_ALLOC(L.count.alloc(L.n, arena));
    SVO_TRY_ALLOC(L.S.alloc(L.n, arena));
    L.dn = n_kept.p;
    if (tiles == 0) {
        SVO_CUDA_TRY(cudaMemsetAsync(n_kept.p, 0, sizeof(uint32_t), st));
        return SVO_OK;
    }
    DevBuf<uint32_t> tn, tf;
    SVO_TRY_ALLOC(tn.alloc(tiles, arena));
    k_brick_keep_count<<<(unsigned)tiles, kBrickThreads, 0, st>>>(b, tn.p);
    SVO_LAUNCH_CHECK("k_brick_keep_count");
    const bool self = tiles <= kSelfScanTiles;
    if (!self) {
        SVO_TRY_ALLOC(tf.alloc(tiles, arena));
        int rc = scan_on_device<uint32_t>(tn.p, tf.p, tiles, n_kept.p, st, arena);
        if (rc) return rc;
    }
    k_brick_keep<<<(unsigned)tiles, kBrickThreads, 0, st>>>(b, tn.p, self ? nullptr : tf.p, L.key.p, src.p, L.mask.p,
                                                            L.count.p, L.S.p, n_kept.p);
    SVO_LAUNCH_CHECK("k_brick_keep");
    return SVO_OK;
}

}  // namespace

int build_from_sorted_device(const uint64_t *d_keys, const uint32_t *d_payload, uint64_t N, int log_side,
                             int log_block, const uint8_t *d_topflag, cudaStream_t st, uint32_t **d_words_out,
                             uint64_t *n_words_out) {
    const int D = log_side;
    if (N >= 0xFFFFFFFFull) return set_error(SVO_ERR_LIMIT, "%llu occupied voxels exceed 2^32-1", (unsigned long long)N);
    BuildArena arena(st);  // declared first: released after every array below
    std::vector<LevelArrays> lv(D + 1);
    auto leaves = [&](uint32_t *words, uint64_t W, uint32_t *err) -> int {
        if (!N) return SVO_OK;
        k_place_leaf_runs<<<blocks_for(lv[1].n), 256, 0, st>>>(lv[1].n, lv[1].dn, lv[1].count.p, lv[1].start.p,
                                                               lv[1].B.p, d_payload, N, words, W, err);
        SVO_LAUNCH_CHECK("k_place_leaf_runs");
        return SVO_OK;
    };
    return build_levels(lv, 0, d_keys, N, D, log_block, d_topflag, arena, st, nullptr, leaves, d_words_out,
                        n_words_out);
}

bool bricks_dense(int log_side, int log_brick) { return 3 * (log_side - log_brick) <= kPyramidBits; }

// The build above bricks whose subtree words (and masks, presence) are arrays
// over all brick codes; place_bricks(places, words, W, err) writes the bricks'
// own words, places.n, .src and the like left to it.
template <typename PlaceBricks>
static int build_pyramid(int base, int D, const uint32_t *words_of, const uint8_t *mask_of, const uint8_t *any_of,
                         int log_block, const uint8_t *d_topflag, BuildArena &arena, cudaStream_t st,
                         const unsigned long long *n_voxels, PlaceBricks place_bricks, uint32_t **d_words_out,
                         uint64_t *n_words_out) {
    if (log_block < D && !any_of && !d_topflag) return set_error(SVO_ERR_INVALID, "build: missing cache-block flags");
    Pyramid p{};
    p.base = base;
    p.top = D;
    p.words_of = words_of;
    p.mask_of = mask_of;
    p.any_of = any_of;
    p.topflag = log_block < D ? d_topflag : nullptr;
    p.log_block = log_block;
    DevBuf<uint64_t> S[kPyramidMax], B[kPyramidMax];
    DevBuf<uint8_t> mask[kPyramidMax], meta[kPyramidMax];
    Report report;  // root's words, voxels (64 bits each), errors
    SVO_CUDA_TRY(report.open(st));
    for (int l = 0; l <= D - base; ++l) {
        const uint64_t cells = 1ull << (3 * (D - base - l));
        SVO_TRY_ALLOC(B[l].alloc(cells, arena));
        p.B[l] = B[l].p;
        if (!l) continue;
        SVO_TRY_ALLOC(S[l].alloc(cells, arena));
        SVO_TRY_ALLOC(mask[l].alloc(cells, arena));
        SVO_TRY_ALLOC(meta[l].alloc(cells, arena));
        p.S[l] = S[l].p;
        p.mask[l] = mask[l].p;
        p.meta[l] = meta[l].p;
    }
    // levels with more than kTopCells children one launch each, the rest in one
    int e = base + 1;
    for (; e <= D && (1ull << (3 * (D - e + 1))) > kTopCells; ++e) {
        const uint64_t cells = 1ull << (3 * (D - e));
        SVO_CUDA_TRY(launch_chained(k_pyramid_up, blocks_for(cells), 256, st, p, e));
    }
    if (e <= D) {
        SVO_CUDA_TRY(launch_chained(k_pyramid_top_up, 1, 512, st, p, e, n_voxels, (uint64_t *)report.device()));
    }
    uint64_t S_root = 0;
    unsigned long long voxels = 0;
    if (D == base) {
        uint32_t s32 = 0;
        SVO_CUDA_TRY(cudaMemcpyAsync(&s32, words_of, sizeof(s32), cudaMemcpyDeviceToHost, st));
        SVO_CUDA_TRY(cudaStreamSynchronize(st));
        S_root = s32;
    } else {
        SVO_CUDA_TRY(report.wait());
        S_root = ((const uint64_t *)report.words())[0];
        voxels = ((const uint64_t *)report.words())[1];
    }
    if (voxels >= 0xFFFFFFFFull) return set_error(SVO_ERR_LIMIT, "%llu occupied voxels exceed 2^32-1", voxels);
    const uint64_t W = 1 + S_root;
    uint32_t *words = nullptr;
    SVO_CUDA_TRY(alloc_words(&words, W, st));
    auto place = [&]() -> int {
        uint32_t *const err = report.device() + 4;
        int c = D;
        while (c > base && (1ull << (3 * (D - c + 1))) <= kTopPlaced) --c;
        k_pyramid_top_down<<<1, (unsigned)kTopPlaced, 0, st>>>(p, c, words, W, err);
        SVO_LAUNCH_CHECK("k_pyramid_top_down");
        for (--c; c >= base; --c) {
            SVO_CUDA_TRY(launch_chained(k_pyramid_down, blocks_for(1ull << (3 * (D - c))), 256, st, p, c, words, W, err));
        }
        BrickPlaces places{};
        places.words_of = words_of;
        places.B = p.B[0];
        int r = place_bricks(places, words, W, err);
        if (r) return r;
        SVO_CUDA_TRY(report.wait());
        if (const uint32_t err_h = report.words()[4]) return set_error(SVO_ERR_DEVICE, "octree build placement check failed (flags %u)", err_h);
        return SVO_OK;
    };
    const int rc = place();
    if (rc) {
        free_words(words, W, st);
        return rc;
    }
    *d_words_out = words;
    *n_words_out = W;
    return SVO_OK;
}

int build_from_bricks_device(const MeshBricks &m, int log_side, int log_block, const uint8_t *d_topflag,
                             cudaStream_t st, uint32_t **d_words_out, uint64_t *n_words_out) {
    constexpr int kBase = 3;
    const int D = log_side;
    BuildArena arena(st);
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((m.n + 7) / 8, 1ull << 20));
    if (bricks_dense(D, kBase)) {
        auto bricks = [&](BrickPlaces places, uint32_t *words, uint64_t W, uint32_t *err) -> int {
            places.src = m.key;
            SVO_CUDA_TRY(launch_chained(k_place_brick8<true>, grid, 256, st, places, m.n, m.bits, m.slot, words, W, err));
            return SVO_OK;
        };
        return build_pyramid(kBase, D, m.words, m.mask, nullptr, log_block, d_topflag, arena, st, m.n_voxels, bricks,
                             d_words_out, n_words_out);
    }
    std::vector<LevelArrays> lv(D + 1);
    DevBuf<uint32_t> src, n_kept;
    LevelArrays &L = lv[kBase];
    const BrickNodes b{m.n, m.key, m.words, m.mask, nullptr};
    int rc = keep_bricks(b, m.n, L, src, n_kept, arena, st);
    if (rc) return rc;
    auto bricks = [&](uint32_t *words, uint64_t W, uint32_t *err) -> int {
        const BrickPlaces places{n_kept.p, src.p, L.key.p, nullptr, L.S.p, L.B.p};
        k_place_brick8<false><<<grid, 256, 0, st>>>(places, 0, m.bits, m.slot, words, W, err);
        SVO_LAUNCH_CHECK("k_place_brick8");
        return SVO_OK;
    };
    return build_levels(lv, kBase, nullptr, 0, D, log_block, d_topflag, arena, st, m.n_voxels, bricks, d_words_out,
                        n_words_out);
}

// The dense build through 16^3 bricks: their bits, the levels above them, and
// every brick's words.  Cache blocks, if several, are at least a brick.
static int build_dense_bricks(const GridGeom &g, int D, uint64_t n_bricks, cudaStream_t st, uint32_t **d_words_out,
                              uint64_t *n_words_out) {
    constexpr int kBase = 4;
    const bool multi_block = g.log_block < D, dense = bricks_dense(D, kBase);
    const uint64_t cells = (uint64_t)g.w * (uint64_t)g.h * (uint64_t)g.d;
    const uint64_t covering = (uint64_t)((g.w + 15) / 16) * (uint64_t)((g.h + 15) / 16) * (uint64_t)((g.d + 15) / 16);
    BuildArena arena(st);
    DevBuf<uint32_t> bits, words_of, list, n_list;
    DevBuf<uint8_t> mask_of, any_of;
    DevBuf<unsigned long long> n_voxels;
    SVO_TRY_ALLOC(bits.alloc(covering * 128, st));
    SVO_TRY_ALLOC(words_of.alloc(n_bricks, arena));
    SVO_TRY_ALLOC(mask_of.alloc(n_bricks, arena));
    // where the cache block is a brick, one with only dropped voxels is a
    // descriptor without children
    const bool any = multi_block && g.log_block == kBase;
    if (any) SVO_TRY_ALLOC(any_of.alloc(n_bricks, arena));
    if (dense) {
        SVO_TRY_ALLOC(list.alloc(covering, arena));
        SVO_TRY_ALLOC(n_list.alloc(1, arena));
        SVO_CUDA_TRY(cudaMemsetAsync(n_list.p, 0, sizeof(uint32_t), st));
    }
    if (cells >= 0xFFFFFFFFull) {  // the voxels may exceed the build's limit
        SVO_TRY_ALLOC(n_voxels.alloc(1, arena));
        SVO_CUDA_TRY(cudaMemsetAsync(n_voxels.p, 0, sizeof(unsigned long long), st));
    }
    const unsigned grid = (unsigned)std::min<uint64_t>(n_bricks, 1ull << 20);
    k_brick_bits<<<grid, kBrickThreads, 0, st>>>(g, n_bricks, bits.p, words_of.p, mask_of.p, any_of.p, list.p,
                                                 n_list.p, n_voxels.p);
    SVO_LAUNCH_CHECK("k_brick_bits");
    // a cache block that is a brick is a node already
    const int log_block = any ? D : g.log_block;
    const uint8_t *const topflag = any ? nullptr : g.topflag;
    const unsigned pgrid = (unsigned)std::min<uint64_t>(covering, 1ull << 14);
    if (dense) {
        auto bricks = [&](BrickPlaces places, uint32_t *words, uint64_t W, uint32_t *err) -> int {
            places.n = n_list.p;
            places.src = list.p;
            SVO_CUDA_TRY(launch_chained(k_place_brick16<true>, pgrid, kBrickThreads, st, g, places, bits.p, words, W, err));
            return SVO_OK;
        };
        return build_pyramid(kBase, D, words_of.p, mask_of.p, any_of.p, log_block, topflag, arena, st, n_voxels.p,
                             bricks, d_words_out, n_words_out);
    }
    std::vector<LevelArrays> lv(D + 1);
    DevBuf<uint32_t> src, n_kept;
    LevelArrays &L = lv[kBase];
    const BrickNodes b{n_bricks, nullptr, words_of.p, mask_of.p, any_of.p};
    int rc = keep_bricks(b, covering, L, src, n_kept, arena, st);
    if (rc) return rc;
    auto bricks = [&](uint32_t *words, uint64_t W, uint32_t *err) -> int {
        const BrickPlaces places{n_kept.p, nullptr, L.key.p, nullptr, L.S.p, L.B.p};
        k_place_brick16<false><<<pgrid, kBrickThreads, 0, st>>>(g, places, bits.p, words, W, err);
        SVO_LAUNCH_CHECK("k_place_brick16");
        return SVO_OK;
    };
    return build_levels(lv, kBase, nullptr, 0, D, log_block, topflag, arena, st, n_voxels.p, bricks, d_words_out,
                        n_words_out);
}

int build_dense_device(const uint32_t *d_grid, int w, int h, int d, int log_side, int log_block, cudaStream_t st,
                       uint32_t **d_words_out, uint64_t *n_words_out) {
    const int D = log_side;
    const int log_brick = D < 4 ? D : 4;
    const uint64_t n_bricks = 1ull << (3 * (D - log_brick));
    const bool multi_block = log_block < D;

    GridGeom g;
    g.grid = d_grid;
    g.w = w;
    g.h = h;
    g.d = d;
    g.log_brick = log_brick;
    g.drop_last_z = ((d & 1) && log_block >= 2) ? 1 : 0;
    g.log_block = log_block;
    g.topflag = nullptr;

    const uint64_t n_blocks = multi_block ? (1ull << (3 * (D - log_block))) : 0;
    if (n_blocks > (1ull << 27))
        return set_error(SVO_ERR_LIMIT, "memory budget gives %llu cache blocks; the GPU build supports at most 2^27",
                         (unsigned long long)n_blocks);
    DevBuf<uint8_t> topflag;
    if (multi_block) {
        SVO_TRY_ALLOC(topflag.alloc(n_blocks, st));
        SVO_CUDA_TRY(cudaMemsetAsync(topflag.p, 0, n_blocks, st));
        g.topflag = topflag.p;
    }
    // Brick keys index 32-bit source arrays; smaller cubes and cache blocks
    // below a brick (budgets of a few KB) take the voxel by voxel form.
    if (D >= 4 && (!multi_block || log_block >= 4) && n_bricks <= 0xFFFFFFFFull)
        return build_dense_bricks(g, D, n_bricks, st, d_words_out, n_words_out);

    // Phase 1: extraction in Morton order.
    DevBuf<uint32_t> bcount;
    DevBuf<uint64_t> boff;
    SVO_TRY_ALLOC(bcount.alloc(n_bricks, st));
    SVO_TRY_ALLOC(boff.alloc(n_bricks, st));
    unsigned grid1 = (unsigned)(n_bricks < (1ull << 20) ? n_bricks : (1ull << 20));
    k_brick_count<<<grid1, kBrickThreads, 0, st>>>(g, n_bricks, bcount.p);
    SVO_LAUNCH_CHECK("k_brick_count");
    uint64_t N = 0;
    int rc = scan_to<uint64_t>(bcount.p, boff.p, n_bricks, &N, st);
    if (rc) return rc;
    if (N >= 0xFFFFFFFFull) return set_error(SVO_ERR_LIMIT, "%llu occupied voxels exceed 2^32-1", (unsigned long long)N);

    DevBuf<uint64_t> lkey;
    DevBuf<uint32_t> lpay;
    SVO_TRY_ALLOC(lkey.alloc(N, st));
    SVO_TRY_ALLOC(lpay.alloc(N, st));
    if (N) {
        k_brick_emit<<<grid1, kBrickThreads, 0, st>>>(g, n_bricks, bcount.p, boff.p, lkey.p, lpay.p);
        SVO_LAUNCH_CHECK("k_brick_emit");
    }
    bcount.release();
    boff.release();

    // Phases 2 and 3.
    return build_from_sorted_device(lkey.p, lpay.p, N, D, log_block, topflag.p, st, d_words_out, n_words_out);
}

}  // namespace svo

// ---- allocation-free build ---------------------------------------------------
//
// svo_octree_build_dense_noalloc: the build above for callers that must not
// allocate device memory at call time.  Its scratch is the file-scope arena
// below (32 MiB, reserved on every device that loads the library until the
// process exits); inputs and the output word buffer come from the caller.
namespace svo {
namespace {

constexpr size_t kNoAllocScratchBytes = 32ull << 20;
constexpr uint64_t kNoAllocMaxVoxels = 1ull << 18;
constexpr int kNoAllocMaxSide = 256;
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) unsigned char g_build_scratch[kNoAllocScratchBytes];

std::mutex g_scratch_mtx;
void *g_scratch_addr[kNoAllocMaxDevices] = {};

// Device address of the arena for the current device.  The first call on a
// device resolves it (cudaGetSymbolAddress) with that device current.
int scratch_for_current_device(unsigned char **out) {
    int dev = 0;
    SVO_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) return set_error(SVO_ERR_LIMIT, "device ordinal %d unsupported", dev);
    std::lock_guard<std::mutex> lock(g_scratch_mtx);
    if (!g_scratch_addr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_build_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(build scratch)");
        g_scratch_addr[dev] = p;
    }
    *out = (unsigned char *)g_scratch_addr[dev];
    return SVO_OK;
}

// Bump allocator over the arena; every call starts from offset 0.
struct Arena {
    unsigned char *base;
    size_t used = 0;
    template <typename T>
    T *take(uint64_t n) {
        size_t bytes = ((size_t)(n ? n : 1) * sizeof(T) + 255) & ~size_t(255);
        if (used + bytes > kNoAllocScratchBytes) return nullptr;
        T *p = (T *)(base + used);
        used += bytes;
        return p;
    }
};

#define SVO_ARENA_TAKE(ptr, T, n)                                                                  \
    T *ptr = arena.take<T>(n);                                                                     \
    if (!ptr) return set_error(SVO_ERR_LIMIT, "build scratch (%zu bytes) exhausted", kNoAllocScratchBytes)

template <typename TO>
int arena_scan(Arena &arena, const uint32_t *in, TO *out, uint64_t n, TO *total_host, cudaStream_t st) {
    size_t mark = arena.used;
    SVO_ARENA_TAKE(scratch, TO, scan_scratch_elems(n));
    SVO_ARENA_TAKE(tot, TO, 1);
    SVO_CUDA_TRY((exclusive_scan<uint32_t, TO>(in, out, n, tot, scratch, st)));
    SVO_CUDA_TRY(cudaMemcpyAsync(total_host, tot, sizeof(TO), cudaMemcpyDeviceToHost, st));
    SVO_CUDA_TRY(cudaStreamSynchronize(st));
    arena.used = mark;
    return SVO_OK;
}

struct ArenaLevel {
    uint64_t n = 0;
    uint64_t *key = nullptr, *S = nullptr, *B = nullptr;
    uint32_t *start = nullptr;
    uint8_t *mask = nullptr, *count = nullptr, *large = nullptr;
};

int build_dense_noalloc(const uint32_t *d_grid, int w, int h, int d, int log_side, int log_block, cudaStream_t st,
                        uint32_t *d_words, uint64_t capacity, uint64_t *n_words_out) {
    Arena arena;
    int rc = scratch_for_current_device(&arena.base);
    if (rc) return rc;
    const int D = log_side;
    const int log_brick = D < 4 ? D : 4;
    const uint64_t n_bricks = 1ull << (3 * (D - log_brick));
    const bool multi_block = log_block < D;
    const uint64_t n_blocks = multi_block ? (1ull << (3 * (D - log_block))) : 0;

    GridGeom g;
    g.grid = d_grid;
    g.w = w;
    g.h = h;
    g.d = d;
    g.log_brick = log_brick;
    g.drop_last_z = ((d & 1) && log_block >= 2) ? 1 : 0;
    g.log_block = log_block;
    g.topflag = nullptr;
    if (multi_block) {
        SVO_ARENA_TAKE(tf, uint8_t, n_blocks);
        SVO_CUDA_TRY(cudaMemsetAsync(tf, 0, n_blocks, st));  // the arena keeps the previous call's bytes
        g.topflag = tf;
    }
    SVO_ARENA_TAKE(bcount, uint32_t, n_bricks);
    SVO_ARENA_TAKE(boff, uint64_t, n_bricks);
    unsigned grid1 = (unsigned)(n_bricks < (1ull << 20) ? n_bricks : (1ull << 20));
    k_brick_count<<<grid1, kBrickThreads, 0, st>>>(g, n_bricks, bcount);
    SVO_LAUNCH_CHECK("k_brick_count");
    uint64_t N = 0;
    rc = arena_scan<uint64_t>(arena, bcount, boff, n_bricks, &N, st);
    if (rc) return rc;
    if (N > kNoAllocMaxVoxels)
        return set_error(SVO_ERR_LIMIT, "%llu occupied voxels exceed the allocation-free build's limit of %llu",
                         (unsigned long long)N, (unsigned long long)kNoAllocMaxVoxels);
    SVO_ARENA_TAKE(lkey, uint64_t, N);
    SVO_ARENA_TAKE(lpay, uint32_t, N);
    if (N) {
        k_brick_emit<<<grid1, kBrickThreads, 0, st>>>(g, n_bricks, bcount, boff, lkey, lpay);
        SVO_LAUNCH_CHECK("k_brick_emit");
    }

    ArenaLevel lv[17];
    uint32_t *leaf_pidx = nullptr;
    const uint64_t *ckey = lkey;
    uint64_t nc = N;
    for (int e = 1; e <= D; ++e) {
        ArenaLevel &L = lv[e];
        SVO_ARENA_TAKE(head, uint32_t, nc);
        SVO_ARENA_TAKE(pidx, uint32_t, nc);
        if (nc) {
            k_heads<<<blocks_for(nc), 256, 0, st>>>(ckey, nc, nullptr, head);
            SVO_LAUNCH_CHECK("k_heads");
        }
        uint32_t np = 0;
        if (multi_block && e == log_block) {
            SVO_ARENA_TAKE(first, uint32_t, n_blocks);
            SVO_ARENA_TAKE(present, uint32_t, n_blocks);
            SVO_ARENA_TAKE(bidx, uint32_t, n_blocks);
            SVO_CUDA_TRY(cudaMemsetAsync(first, 0xFF, n_blocks * sizeof(uint32_t), st));
            if (nc) k_block_first<<<blocks_for(nc), 256, 0, st>>>(ckey, nc, nullptr, head, first);
            k_block_present<<<blocks_for(n_blocks), 256, 0, st>>>(first, g.topflag, n_blocks, present);
            SVO_LAUNCH_CHECK("k_block_present");
            rc = arena_scan<uint32_t>(arena, present, bidx, n_blocks, &np, st);
            if (rc) return rc;
            L.n = np;
            SVO_ARENA_TAKE(key, uint64_t, np);
            SVO_ARENA_TAKE(start, uint32_t, np);
            L.key = key;
            L.start = start;
            k_block_parents<<<blocks_for(n_blocks), 256, 0, st>>>(first, present, bidx, n_blocks, nc, nullptr, L.key,
                                                                  L.start);
            if (nc) k_child_pidx_from_blocks<<<blocks_for(nc), 256, 0, st>>>(ckey, nc, nullptr, bidx, pidx);
            SVO_LAUNCH_CHECK("k_child_pidx_from_blocks");
        } else {
            rc = arena_scan<uint32_t>(arena, head, pidx, nc, &np, st);
            if (rc) return rc;
            L.n = np;
            SVO_ARENA_TAKE(key, uint64_t, np);
            SVO_ARENA_TAKE(start, uint32_t, np);
            L.key = key;
            L.start = start;
            if (nc) {
                k_parents_from_heads<<<blocks_for(nc), 256, 0, st>>>(ckey, nc, nullptr, head, pidx, L.key, L.start);
                k_child_pidx_from_heads<<<blocks_for(nc), 256, 0, st>>>(head, nc, nullptr, pidx);
                SVO_LAUNCH_CHECK("k_child_pidx_from_heads");
            }
        }
        if (e == D && L.n == 0) {
            L.n = 1;
            SVO_ARENA_TAKE(key, uint64_t, 1);
            SVO_ARENA_TAKE(start, uint32_t, 1);
            L.key = key;
            L.start = start;
            SVO_CUDA_TRY(cudaMemsetAsync(L.key, 0, sizeof(uint64_t), st));
            SVO_CUDA_TRY(cudaMemsetAsync(L.start, 0, sizeof(uint32_t), st));
        }
        SVO_ARENA_TAKE(mask, uint8_t, L.n);
        SVO_ARENA_TAKE(count, uint8_t, L.n);
        L.mask = mask;
        L.count = count;
        k_parent_masks<<<blocks_for(L.n), 256, 0, st>>>(L.key, L.start, L.n, nullptr, ckey, nc, nullptr, L.mask,
                                                        L.count);
        SVO_LAUNCH_CHECK("k_parent_masks");
        if (e == 1) leaf_pidx = pidx;
        ckey = L.key;
        nc = L.n;
    }
    for (int e = 1; e <= D; ++e) {
        ArenaLevel &L = lv[e];
        SVO_ARENA_TAKE(S, uint64_t, L.n);
        SVO_ARENA_TAKE(large, uint8_t, L.n);
        L.S = S;
        L.large = large;
        k_subtree<<<blocks_for(L.n), 256, 0, st>>>(L.n, nullptr, L.count, L.start, e > 1 ? lv[e - 1].S : nullptr, e == 1,
                                                  L.S, L.large);
        SVO_LAUNCH_CHECK("k_subtree");
    }
    uint64_t S_root = 0;
    SVO_CUDA_TRY(cudaMemcpyAsync(&S_root, lv[D].S, sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    SVO_CUDA_TRY(cudaStreamSynchronize(st));
    const uint64_t W = 1 + S_root;
    *n_words_out = W;
    if (W > capacity)
        return set_error(SVO_ERR_LIMIT, "octree needs %llu words; the output buffer holds %llu",
                         (unsigned long long)W, (unsigned long long)capacity);
    SVO_ARENA_TAKE(err, uint32_t, 1);
    SVO_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(uint32_t), st));
    SVO_ARENA_TAKE(rootB, uint64_t, 1);
    lv[D].B = rootB;
    k_root_word<<<1, 1, 0, st>>>(lv[D].mask, lv[D].large, D == 1, lv[D].B, d_words);
    for (int e = D; e >= 2; --e) {
        ArenaLevel &P = lv[e];
        ArenaLevel &C = lv[e - 1];
        SVO_ARENA_TAKE(cB, uint64_t, C.n);
        C.B = cB;
        k_place<<<blocks_for(P.n), 256, 0, st>>>(P.n, nullptr, P.count, P.start, P.large, P.B, C.S, C.mask, C.large,
                                                e - 1 == 1, C.B, d_words, W, err);
        SVO_LAUNCH_CHECK("k_place");
    }
    if (N) {
        k_place_leaves<<<blocks_for(N), 256, 0, st>>>(N, leaf_pidx, lv[1].n, nullptr, lv[1].start, lv[1].B, lpay, d_words, W,
                                                      err);
        SVO_LAUNCH_CHECK("k_place_leaves");
    }
    uint32_t err_h = 0;
    SVO_CUDA_TRY(cudaMemcpyAsync(&err_h, err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    SVO_CUDA_TRY(cudaStreamSynchronize(st));
    if (err_h) return set_error(SVO_ERR_DEVICE, "octree build placement check failed (flags %u)", err_h);
    return SVO_OK;
}

}  // namespace
}  // namespace svo

extern "C" int svo_octree_build_dense_noalloc(const uint32_t *d_grid, int w, int h, int d, uint64_t mem,
                                              uint32_t *d_words, uint64_t capacity, uint64_t *n_words,
                                              float center[3], svo_stream stream) {
    using namespace svo;
    if (!d_grid || !d_words || !n_words || !center || w <= 0 || h <= 0 || d <= 0)
        return set_error(SVO_ERR_INVALID, "bad arguments");
    // checked before the doubling below, which would overflow past 2^30
    if (w > kNoAllocMaxSide || h > kNoAllocMaxSide || d > kNoAllocMaxSide)
        return set_error(SVO_ERR_LIMIT, "grid %d x %d x %d exceeds the allocation-free build's limit of side %d", w,
                         h, d, kNoAllocMaxSide);
    int side = 1;
    while (side < w || side < h || side < d) side *= 2;
    if (side < 2) return set_error(SVO_ERR_INVALID, "virtual side %d below 2 (the reference recurses forever)", side);
    int lb = cache_block_log2(w, h, d, mem, 4);
    if (lb < 1) return set_error(SVO_ERR_MEMORY, "memory budget %llu admits no cache block", (unsigned long long)mem);
    int log_side = 0;
    while ((1 << log_side) < side) ++log_side;
    int rc = build_dense_noalloc(d_grid, w, h, d, log_side, lb, (cudaStream_t)stream, d_words, capacity, n_words);
    if (rc) {
        // an error can leave earlier launches queued; they still write to the
        // shared arena, so wait for them before returning (the error already
        // recorded stays the one reported)
        cudaStreamSynchronize((cudaStream_t)stream);
        return rc;
    }
    center[0] = (float)w * 0.5f / (float)side;
    center[1] = (float)h * 0.5f / (float)side;
    center[2] = (float)d * 0.5f / (float)side;
    return SVO_OK;
}
