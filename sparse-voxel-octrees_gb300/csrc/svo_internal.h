// svo_internal.h — host-side internals shared by the library's translation units.
#pragma once

#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "svo.h"

// The opaque handle behind svo_octree*.
struct svo_octree {
    uint32_t *d_words = nullptr;  // resident octree words (HBM), the error word behind them
    uint64_t n_words = 0;
    bool plain_words = false;  // from cudaMalloc, not the library's pool
    float center[3] = {0.0f, 0.0f, 0.0f};
    int device = 0;
    int levels = 0;  // descriptor levels, 0: not known
    uint32_t *d_status = nullptr;  // device error word, behind the words: bit 0 = a ray ended with kFault
    int index_bits = 32;  // 64: svo_trace uses 64-bit word indices even when n_words fits 32 bits

    // Descriptor table of the table traversal (octree_table.cu), built by the
    // first trace call that can use it; a cache of the immutable words.
    mutable uint4 *d_tab = nullptr;
    mutable uint64_t n_tab = 0;
    mutable std::atomic<int> tab_state{0};  // 0 not built yet, 1 built, -1 the octree does not qualify
    bool use_table = true;
    mutable std::mutex tab_mtx;

    // Host-buffer pipeline of svo_trace_host and svo_trace_image_host: one
    // device staging arena split into kStageBuffers buffers, a copy-in and a
    // copy-out stream, one trace stream per buffer, and per-buffer events
    // (inputs landed, trace done, outputs copied).
    static constexpr int kStageBuffers = 4;  // stage_used has one flag per buffer
    std::mutex staging_mtx;
    void *stage_dev = nullptr;
    size_t stage_dev_bytes = 0;
    uint64_t stage_cap = 0;       // rays per staging buffer (the arena's layout)
    uint64_t stage_seq = 0;       // chunks enqueued so far: chunk k uses buffer k % kStageBuffers
    bool stage_used[4] = {};      // the buffer holds an earlier chunk (its events are waited on)
    bool stage_pending = false;   // enqueued work not yet drained (svo_octree_synchronize)
    cudaStream_t copy_in = nullptr, copy_out = nullptr;
    cudaStream_t stage_trace[kStageBuffers] = {};
    cudaEvent_t stage_in[kStageBuffers] = {}, stage_traced[kStageBuffers] = {}, stage_out[kStageBuffers] = {};
};

namespace svo {

// Octrees above 2^32-1 words need 64-bit word indices: far offsets then carry
// bits above 32 in the descriptor's top 14 bits (VoxelOctree.cpp:190-194).
constexpr uint64_t kMaxNarrowWords = 0xFFFFFFFFull;
inline bool wide_octree(const svo_octree *o) { return o->n_words > kMaxNarrowWords; }

// Records a formatted message for svo_last_error() and returns `code`.
int set_error(int code, const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *what);
void clear_error();

#define SVO_CUDA_TRY(call)                                   \
    do {                                                     \
        cudaError_t _e = (call);                             \
        if (_e != cudaSuccess) return ::svo::cuda_fail(_e, #call); \
    } while (0)

// LZ4 block format (independent blocks; decoder accepts history before pos0).
size_t lz4_compress_bound(size_t n);
size_t lz4_compress_block(const uint8_t *src, size_t n, uint8_t *dst, size_t cap);
int lz4_decompress_block(const uint8_t *src, size_t src_len, uint8_t *out, size_t pos0, size_t out_len);

// Stream-ordered scratch from the library's per-device pool (mem_pool.cpp);
// release with cudaFreeAsync.
cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t st);

// Memory that a handle keeps, from a pool of its own or, when large, the
// driver's; release with handle_free (and the same size) once nothing on the
// device uses it any more.
cudaError_t handle_alloc(void **p, size_t bytes, cudaStream_t st);
cudaError_t handle_free(void *p, size_t bytes, cudaStream_t st);

// The same for memory of the current device that its streams may still use:
// waits for the device first, and keeps the memory aside where that is refused.
struct HandleMemory {
    void *p;
    size_t bytes;
    bool plain;  // from cudaMalloc
};
void handle_retire(const HandleMemory *blocks, int n);
size_t words_bytes(uint64_t n);  // of alloc_words

// An octree's words from that pool, with the handle's zeroed error word behind
// them, at status_offset(n) words.  plain: from cudaMalloc instead, for words
// that were so before the pool: such memory can be shared with other processes
// and devices.
constexpr uint64_t kStatusWords = 32;
inline uint64_t status_offset(uint64_t n_words) { return (n_words + 31) / 32 * 32; }
cudaError_t alloc_words(uint32_t **words, uint64_t n, cudaStream_t st, bool plain = false);
void free_words(uint32_t *words, uint64_t n, cudaStream_t st, bool plain = false);  // of alloc_words, or null

// A non-blocking stream per device, shared by the library's own work.
cudaError_t library_stream(cudaStream_t *out);

// Page-locked memory that the device reads and writes in place, with a stream,
// for host calls too small for copies to pay (mem_pool.cpp).  host_slot_take
// returns null when none can be had; a slot is idle on the device when it is
// given back.
constexpr size_t kHostSlotBytes = 1u << 20;
struct HostSlot {
    int device;
    char *host, *dev;  // the same memory
    cudaStream_t st;
    cudaEvent_t order;  // to put the stream behind another's work
};
HostSlot *host_slot_take();
void host_slot_give(HostSlot *slot);

// A few words that kernels of a call report to the host.  They lie in a host
// slot's page-locked memory, which the kernels write themselves, so that the
// host only waits for the stream.  A copy of a few bytes to pageable memory
// costs 10 us more: the octree, table and first view of a 200x131x177 volume,
// four such waits, took 207 us with copies and 170 without.  Where no slot can
// be had they lie on the device and wait() copies them.
class Report {
  public:
    static constexpr uint32_t kWords = 64;
    Report() = default;
    Report(const Report &) = delete;
    Report &operator=(const Report &) = delete;
    ~Report();
    cudaError_t open(cudaStream_t st);  // the words are zero
    // the words, for a kernel that is launched next on the stream
    uint32_t *device() {
        busy_ = true;
        return dev_;
    }
    cudaError_t wait();  // for the stream; words() then holds what was reported
    const uint32_t *words() const { return slot_ ? (const uint32_t *)slot_->host : copy_; }

  private:
    HostSlot *slot_ = nullptr;
    uint32_t *dev_ = nullptr;
    cudaStream_t st_ = nullptr;
    bool busy_ = false;
    uint32_t copy_[kWords] = {};
};

// VoxelData::init cache-block search (VoxelData.cpp:211-244): log2 of the
// cache-block edge, or -1 when no partition fits `mem`.
int cache_block_log2(int w, int h, int d, uint64_t mem, uint64_t cell_cost);

// GPU build from a device-resident dense grid (build.cu).  On success the
// caller owns *d_words (make_handle, or free_words).
int build_dense_device(const uint32_t *d_grid, int w, int h, int d, int log_side, int log_block, cudaStream_t st,
                       uint32_t **d_words, uint64_t *n_words);

// Phases 2-3 of the build (build.cu) from voxels already in ascending Morton
// order: d_keys are Morton codes over a 2^log_side cube, d_payload the leaf
// words.  d_topflag (one byte per cache block, Morton-indexed) is required
// when log_block < log_side and marks blocks that exist without children.
int build_from_sorted_device(const uint64_t *d_keys, const uint32_t *d_payload, uint64_t n, int log_side,
                             int log_block, const uint8_t *d_topflag, cudaStream_t st, uint32_t **d_words,
                             uint64_t *n_words);

// The same from 8^3 bricks in ascending Morton order (brick.cuh): per brick its
// key (the Morton code of the brick), 16 words of occupancy bits and 512 words
// holding its voxels in Morton order; and per brick, or with bricks_dense(
// log_side, 3) per brick code of the whole cube, the subtree's words (0 where
// there is no voxel) and the node's mask.  n_voxels: the voxels' total, or
// null where it is known to be below 2^32-1.  log_block is 4 or more, or
// log_side.
struct MeshBricks {
    uint64_t n;
    const uint32_t *key, *words;
    const uint8_t *mask;
    const uint32_t *bits, *slot;
    const unsigned long long *n_voxels;
};
bool bricks_dense(int log_side, int log_brick);
int build_from_bricks_device(const MeshBricks &m, int log_side, int log_block, const uint8_t *d_topflag,
                             cudaStream_t st, uint32_t **d_words, uint64_t *n_words);

// The .voxel build streamed in z slabs of about slab_bytes (voxel_stream.cu);
// fp is positioned after the 12-byte header.
int build_voxel_file_streamed(FILE *fp, int w, int h, int d, uint64_t mem, uint64_t slab_bytes, cudaStream_t st,
                              uint32_t **d_words, uint64_t *n_words, float center[3]);

// Trace launchers (trace.cu).  status: null for the handle's error word, else
// the word that gets this call's flags and those the handle's word holds.
int launch_trace(const svo_octree *oct, const float *d_rays, uint64_t n, float ray_scale, const float light[3],
                 const svo_trace_out &out, cudaStream_t st, uint32_t *status = nullptr);
int launch_trace_image(const svo_octree *oct, const float *d_rays, uint32_t width, uint32_t height, float ray_scale,
                       const float light[3], const svo_trace_out &out, cudaStream_t st,
                       uint32_t *status = nullptr);
int launch_count_loads(const svo_octree *oct, const float *d_rays, uint64_t n, float ray_scale, uint32_t *loads,
                       cudaStream_t st);

// Creates a handle around device words from alloc_words, complete on the
// device (takes ownership).
// levels: the built cube's descriptor levels, or 0 where they are not known
int make_handle(uint32_t *d_words, uint64_t n_words, const float center[3], svo_octree **out, int levels = 0);

// The handle's descriptor table (octree_table.cu), built on first use; null
// when the octree does not qualify (over 2^32-1 words, or a reachable node
// that fails the checks), when the table is switched off, or while `caller`
// is being captured into a graph.  Synchronous the first time.
const uint4 *octree_table(const svo_octree *oct, cudaStream_t caller);

}  // namespace svo
