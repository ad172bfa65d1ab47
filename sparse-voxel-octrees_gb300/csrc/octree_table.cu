// octree_table.cu — builds an octree handle's descriptor table, the structure
// the table traversal (ray_step_tab) walks instead of decoding relative and
// far offsets with bounds checks at every PUSH.
//
// The traversal needs a node's internal children at consecutive entries, in
// block order, and nothing else of the order.  In the word array they are
// consecutive descriptors already, so the table holds the top kTopLevels
// levels breadth first (the batched kernels' shared-memory caches copy the
// first entries) and every deeper node in word order:
//   1. k_table_top: the top levels, one CTA;
//   2. k_table_expand, a launch per level, no host round trip: every node of
//      the level passes table_node's checks (octree_table.cuh), marks its
//      internal children in a bitmap over the words and appends them to the
//      node list, in any order;
//   3. k_table_tiles, k_table_rank: the bitmap's prefix counts, which are the
//      entries' positions;
//   4. k_table_entries: one pass over the words writes every entry.
// A node reached twice, one between a far block's slots, more nodes than the
// list holds (a quarter of the words) or more than kWordOrderMost words leave
// that to the breadth-first form below, which needs a scan and a host round
// trip per level and keeps shared nodes apart:
//   1. k_table_count: per node of the level, table_node's checks and its
//      internal-child count;
//   2. an exclusive scan of the counts gives each node's first child in the
//      next level;
//   3. k_table_children: the next level's node words (block start + j * stride
//      for a node's j-th internal child);
//   4. k_table_write, once all levels are known: the entries.
// A failed check anywhere, a level past 22 or more entries than words leaves
// the handle without a table.  The table costs 16 bytes per node, about 2
// bytes per octree word on the benchmark scenes.
//
// Measured, first call to ready table (us), word order against breadth first:
// 49 and 309 (10,000 words), 70 and 413 (1.8 M), 140 and 492 (14 M), 458 and 706
// (63 M), 759 and 833 (113 M), 3,240 and 2,100 (490 M: the list's scattered marks
// and the pass over all words then cost more than the round trips).  The
// table of a 200x131x177 volume took 118 without chained launches (chain.cuh),
// 92 with them, 83 with the levels known, and 65 since the kernels write what
// the host waits for into its own memory.
// Traces run at the same speed over either order (within 0.5% on nine
// workloads).
#include <algorithm>
#include <cstring>
#include <memory>
#include <vector>

#include "chain.cuh"
#include "octree_table.cuh"
#include "scan.cuh"
#include "svo_internal.h"

namespace svo {
namespace {

// ---- breadth first -----------------------------------------------------------------

__global__ void __launch_bounds__(256) k_table_count(const uint32_t *__restrict__ words, uint32_t n_words,
                                                     const uint32_t *__restrict__ level, uint32_t n, int L,
                                                     uint32_t *__restrict__ n_int, uint32_t *__restrict__ err) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t cb, stride, k;
    if (!table_node(words, n_words, level[i], L, cb, stride, k)) {
        atomicOr(err, 1u);
        k = 0;
    }
    n_int[i] = k;
}

__global__ void __launch_bounds__(256) k_table_children(const uint32_t *__restrict__ words, uint32_t n_words,
                                                        const uint32_t *__restrict__ level, uint32_t n, int L,
                                                        const uint32_t *__restrict__ first, uint32_t *__restrict__ next) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t cb, stride, k;
    if (!table_node(words, n_words, level[i], L, cb, stride, k)) return;
    const uint32_t o = first[i];
    for (uint32_t j = 0; j < k; ++j) next[o + j] = cb + j * stride;
}

__global__ void __launch_bounds__(256) k_table_write(const uint32_t *__restrict__ words, uint32_t n_words,
                                                     const uint32_t *__restrict__ level, uint32_t n, int L,
                                                     const uint32_t *__restrict__ first, uint32_t next_base,
                                                     uint4 *__restrict__ entries) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t d = level[i];
    uint32_t cb, stride, k;
    table_node(words, n_words, d, L, cb, stride, k);
    entries[i] = make_uint4(words[d], next_base + first[i], cb, 0u);
}

// ---- word order --------------------------------------------------------------------

constexpr int kTopLevels = 4;        // breadth first: at most 1 + 8 + 64 + 512 nodes
constexpr uint64_t kWordOrderMost = 1ull << 27;
constexpr int kTopNodes = 585;
constexpr int kTopThreads = 512;

struct WordOrder {
    const uint32_t *words;
    uint32_t n_words;
    uint32_t *list;   // the deeper nodes' words, level by level
    uint32_t cap;
    uint32_t *bits;   // one per word: the descriptor of a deeper node
    uint32_t *rank;   // per 32 words: deeper nodes before them
    uint32_t *tile;   // per kRankTile words of `bits`: their nodes
    uint32_t *top;    // top nodes: word, first child's entry (last top level: none yet)
    uint32_t *ctl;
};
// ctl: list entries, error flags, top nodes, top nodes above the last top
// level, then per level the list's length after it and the CTAs done with it
constexpr int kCtlTail = 0, kCtlErr = 1, kCtlTop = 2, kCtlInner = 3, kCtlEnd = 4,
              kCtlDone = kCtlEnd + kTableMaxParentLevel + 4, kCtlWords = kCtlDone + kTableMaxParentLevel + 4;
constexpr uint32_t kErrBad = 1, kErrFull = 2, kErrOrder = 4;
constexpr int kRankItems = 8, kRankTile = kScanThreads * kRankItems;
constexpr uint64_t kRankSelf = 1024;  // tiles up to which each sums those before it itself

// Marks the k internal children of a child block in the bitmap.
__device__ __forceinline__ void mark_children(const WordOrder &t, uint32_t cb, uint32_t stride, uint32_t k) {
    const uint64_t m = (stride == 1 ? (1ull << k) - 1 : 0x5555ull & ((1ull << (2 * k)) - 1)) << (cb & 31);
    atomicOr(t.bits + (cb >> 5), (uint32_t)m);
    if (m >> 32) atomicOr(t.bits + (cb >> 5) + 1, (uint32_t)(m >> 32));
}

__device__ __forceinline__ uint32_t rank_of(const WordOrder &t, uint32_t w) {
    return t.rank[w >> 5] + (uint32_t)__popc(t.bits[w >> 5] & ((1u << (w & 31)) - 1u));
}

__global__ void __launch_bounds__(kTopThreads) k_table_top(WordOrder t) {
    __shared__ uint32_t node[kTopNodes], wsum[kTopThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) node[0] = 0;
    uint32_t begin = 0, end = 1;
    for (int L = 0; L < kTopLevels; ++L) {
        __syncthreads();
        const bool live = begin + threadIdx.x < end;
        const uint32_t me = live ? node[begin + threadIdx.x] : 0u;
        uint32_t cb = 0, stride = 1, k = 0;
        if (live && !table_node(t.words, t.n_words, me, L, cb, stride, k)) {
            atomicOr(&t.ctl[kCtlErr], kErrBad);
            k = 0;
        }
        const uint32_t incl = warp_incl_scan(k);
        if (lane == 31) wsum[wid] = incl;
        __syncthreads();
        uint32_t off = incl - k, total = 0;
        for (int w = 0; w < kTopThreads / 32; ++w) {
            if (w < wid) off += wsum[w];
            total += wsum[w];
        }
        const bool last = L == kTopLevels - 1;
        if (live) {
            t.top[2 * (begin + threadIdx.x)] = me;
            t.top[2 * (begin + threadIdx.x) + 1] = end + off;
            if (last && k) mark_children(t, cb, stride, k);
            for (uint32_t j = 0; j < k; ++j) (last ? t.list : node + end)[off + j] = cb + j * stride;
        }
        if (last) {
            if (threadIdx.x == 0) {
                t.ctl[kCtlTop] = end;
                t.ctl[kCtlInner] = begin;
                t.ctl[kCtlTail] = total;
                t.ctl[kCtlEnd + kTopLevels] = total;
            }
        } else {
            begin = end;
            end += total;
        }
    }
}

// Level L's nodes, list[length(L - 1) .. length(L)).  The last CTA to finish
// notes the list's length for the next level; no CTA waits for another.
__global__ void __launch_bounds__(256) k_table_expand(WordOrder t, int L) {
    chain_begin();
    // after an error the list may hold places that were never written (the
    // whole CTA decides: another one of this launch may be setting the flag)
    if (__syncthreads_or(t.ctl[kCtlErr] != 0)) return;
    __shared__ uint32_t base;
    const uint32_t begin = L > kTopLevels ? t.ctl[kCtlEnd + L - 1] : 0u, end = min(t.ctl[kCtlEnd + L], t.cap);
    for (uint32_t i0 = begin + blockIdx.x * blockDim.x; i0 < end; i0 += gridDim.x * blockDim.x) {
        const uint32_t i = i0 + threadIdx.x;
        uint32_t cb = 0, stride = 1, k = 0, total;
        if (i < end && !table_node(t.words, t.n_words, t.list[i], L, cb, stride, k)) {
            atomicOr(&t.ctl[kCtlErr], kErrBad);
            k = 0;
        }
        if (!__syncthreads_or((int)k)) continue;
        const uint32_t off = block_excl_scan<uint32_t>(k, &total);
        // one reservation per CTA: the list's length is one address
        if (threadIdx.x == 0) base = atomicAdd(&t.ctl[kCtlTail], total);
        __syncthreads();
        const uint32_t at = base + off;
        if (!k) continue;
        if (at > t.cap || k > t.cap - at) {
            atomicOr(&t.ctl[kCtlErr], kErrFull);
            continue;
        }
        mark_children(t, cb, stride, k);
        for (uint32_t j = 0; j < k; ++j) t.list[at + j] = cb + j * stride;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&t.ctl[kCtlDone + L], 1u) == gridDim.x - 1)
        t.ctl[kCtlEnd + L + 1] = atomicAdd(&t.ctl[kCtlTail], 0u);
}

__global__ void __launch_bounds__(kScanThreads) k_table_tiles(WordOrder t, uint64_t n) {
    chain_begin();
    const uint64_t i0 = (uint64_t)blockIdx.x * kRankTile + (uint64_t)threadIdx.x * kRankItems;
    uint32_t c = 0, total;
    for (int k = 0; k < kRankItems; ++k)
        if (i0 + k < n) c += (uint32_t)__popc(t.bits[i0 + k]);
    block_excl_scan<uint32_t>(c, &total);
    if (threadIdx.x == 0) t.tile[blockIdx.x] = total;
}

// first: the tiles' scan, or null: this tile adds up those before it.  Reports
// ctl to the host, and as its last word the bitmap's total.
__global__ void __launch_bounds__(kScanThreads) k_table_rank(WordOrder t, uint64_t n, const uint32_t *first,
                                                             uint32_t *__restrict__ report) {
    chain_begin();
    uint32_t before = 0, total;
    if (first) {
        before = first[blockIdx.x];
    } else {
        uint32_t c = 0;
        for (uint32_t i = threadIdx.x; i < blockIdx.x; i += kScanThreads) c += t.tile[i];
        block_excl_scan<uint32_t>(c, &before);
    }
    const uint64_t i0 = (uint64_t)blockIdx.x * kRankTile + (uint64_t)threadIdx.x * kRankItems;
    uint32_t c = 0, own[kRankItems];
    for (int k = 0; k < kRankItems; ++k) {
        own[k] = i0 + k < n ? (uint32_t)__popc(t.bits[i0 + k]) : 0u;
        c += own[k];
    }
    uint32_t at = before + block_excl_scan<uint32_t>(c, &total);
    for (int k = 0; k < kRankItems; ++k) {
        if (i0 + k < n) t.rank[i0 + k] = at;
        at += own[k];
    }
    if (blockIdx.x == 0 && threadIdx.x < kCtlWords - (first ? 0 : 1)) report[threadIdx.x] = t.ctl[threadIdx.x];
    if (!first && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) report[kCtlWords - 1] = before + total;
}

// The entry of a child block's first internal child.  A far block's children
// are consecutive entries only if the far words between them are no
// descriptors.
__device__ __forceinline__ uint32_t child_entry(const WordOrder &t, uint32_t n_top, uint32_t cb, uint32_t stride,
                                                uint32_t k, uint32_t *err) {
    if (!k) return 0u;
    if (stride == 2)
        for (uint32_t f = cb + 1; f < cb + 2 * k - 1; f += 2)
            if ((t.bits[f >> 5] >> (f & 31)) & 1u) atomicOr(err, kErrOrder);
    return n_top + rank_of(t, cb);
}

__global__ void __launch_bounds__(256) k_table_entries(WordOrder t, uint4 *__restrict__ tab, uint32_t *__restrict__ err) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n_top = t.ctl[kCtlTop];
    if (i < n_top) {  // table_node has passed for every node here
        uint32_t cb, stride, k, first = t.top[2 * i + 1];
        table_node(t.words, t.n_words, t.top[2 * i], 0, cb, stride, k);
        if (i >= t.ctl[kCtlInner]) first = child_entry(t, n_top, cb, stride, k, err);
        tab[i] = make_uint4(t.words[t.top[2 * i]], first, cb, 0u);
    }
    if (i >= t.n_words || !((t.bits[i >> 5] >> (i & 31)) & 1u)) return;
    uint32_t cb, stride, k;
    table_node(t.words, t.n_words, (uint32_t)i, 0, cb, stride, k);
    tab[n_top + rank_of(t, (uint32_t)i)] = make_uint4(t.words[i], child_entry(t, n_top, cb, stride, k, err), cb, 0u);
}

struct Scratch {
    void *p = nullptr;
    cudaStream_t st = nullptr;
    Scratch() = default;
    Scratch(const Scratch &) = delete;
    Scratch &operator=(const Scratch &) = delete;
    cudaError_t alloc(size_t bytes, cudaStream_t s) {
        st = s;
        return scratch_alloc(&p, bytes ? bytes : 4, s);
    }
    ~Scratch() {
        if (p) cudaFreeAsync(p, st);
    }
};

inline unsigned grid_for(uint64_t n) { return (unsigned)((n + 255) / 256); }

// The table in word order; *tab stays null when it cannot be had this way.
int build_word_order(const uint32_t *d_words, uint64_t n_words, int levels, cudaStream_t st, uint4 **tab,
                     uint64_t *n_tab) {
    *tab = nullptr;
    // a node list as long as the words where that is little memory, else a
    // quarter of them (about an eighth are nodes on the benchmark scenes)
    constexpr uint64_t kWholeList = 1ull << 24;
    const uint64_t nb = (n_words + 31) / 32, tiles = (nb + kRankTile - 1) / kRankTile;
    const uint64_t cap = std::max<uint64_t>(n_words <= kWholeList ? n_words : n_words / 4, 8 * kTopNodes);
    const bool self = tiles <= kRankSelf;
    auto round4 = [](uint64_t n) { return (n + 3) & ~uint64_t(3); };
    // one block: zeroed ctl and bits (with one more word, for a mark that
    // reaches past the last), then the rest
    const uint64_t o_bits = round4(kCtlWords), o_rank = o_bits + round4(nb + 1), o_tile = o_rank + round4(nb),
                   o_first = o_tile + round4(tiles), o_scan = o_first + (self ? 0 : round4(tiles)),
                   o_top = o_scan + round4(scan_scratch_elems(tiles)), o_list = o_top + round4(2 * kTopNodes);
    Scratch mem;
    SVO_CUDA_TRY(mem.alloc((size_t)(o_list + cap) * sizeof(uint32_t), st));
    uint32_t *const m = (uint32_t *)mem.p;
    WordOrder t;
    t.words = d_words;
    t.n_words = (uint32_t)n_words;
    t.ctl = m;
    t.bits = m + o_bits;
    t.rank = m + o_rank;
    t.tile = m + o_tile;
    t.top = m + o_top;
    t.list = m + o_list;
    t.cap = (uint32_t)cap;
    uint32_t *const first = self ? nullptr : m + o_first;
    SVO_CUDA_TRY(cudaMemsetAsync(m, 0, (size_t)o_rank * sizeof(uint32_t), st));
    k_table_top<<<1, kTopThreads, 0, st>>>(t);
    SVO_CUDA_TRY(cudaGetLastError());
    // a built cube's levels, or twelve (a 4096^3 cube's), before the host looks,
    // and if they end there the ranks are there too; an empty level costs 3 us
    const int expect = levels > kTopLevels ? levels : levels ? kTopLevels + 1 : 12;
    static_assert(kCtlWords <= Report::kWords && kCtlWords <= kScanThreads, "one report");
    Report report;
    SVO_CUDA_TRY(report.open(st));
    uint32_t h[kCtlWords];
    uint32_t n = 0;
    for (int L = kTopLevels;;) {
        const int to = std::min(L == kTopLevels ? expect : L + 6, kTableMaxParentLevel + 2);
        for (; L < to; ++L) {
            const uint64_t most = L < 8 ? std::min<uint64_t>(cap, 1ull << (3 * L)) : cap;
            SVO_CUDA_TRY(launch_chained(k_table_expand, (unsigned)std::min<uint64_t>((most + 255) / 256, 152 * 8), 256, st,
                                        t, L));
        }
        SVO_CUDA_TRY(launch_chained(k_table_tiles, (unsigned)tiles, kScanThreads, st, t, nb));
        if (!self)
            SVO_CUDA_TRY((exclusive_scan<uint32_t, uint32_t>(t.tile, first, tiles, t.ctl + kCtlWords - 1, m + o_scan, st)));
        SVO_CUDA_TRY(launch_chained(k_table_rank, (unsigned)tiles, kScanThreads, st, t, nb, first,
                                    report.device()));
        SVO_CUDA_TRY(report.wait());
        std::memcpy(h, report.words(), sizeof(h));
        if (h[kCtlErr]) return SVO_OK;
        if (h[kCtlEnd + L] == h[kCtlEnd + L - 1]) break;  // the last level expanded added nothing
        if (L >= kTableMaxParentLevel + 2) return SVO_OK;
    }
    if (h[kCtlWords - 1] != h[kCtlTail]) return SVO_OK;  // a node reached twice
    n = h[kCtlTop] + h[kCtlTail];
    uint4 *e = nullptr;
    SVO_CUDA_TRY(handle_alloc((void **)&e, (size_t)n * sizeof(uint4), st));
    k_table_entries<<<grid_for(std::max<uint64_t>(n_words, kTopNodes)), 256, 0, st>>>(t, e, report.device() + kCtlErr);
    cudaError_t er = cudaGetLastError();
    if (er == cudaSuccess) er = report.wait();
    if (er != cudaSuccess || report.words()[kCtlErr]) {
        handle_free(e, (size_t)n * sizeof(uint4), st);
        return er != cudaSuccess ? cuda_fail(er, "descriptor table") : SVO_OK;
    }
    *tab = e;
    *n_tab = n;
    return SVO_OK;
}

// Builds the table on `st` and waits for it.  Returns SVO_OK with *tab set
// (handle_alloc'd, n_tab entries) or with *tab = nullptr when the octree does
// not qualify; an error code only for CUDA failures.
int build_table(const uint32_t *d_words, uint64_t n_words, int levels, cudaStream_t st, uint4 **tab, uint64_t *n_tab) {
    *tab = nullptr;
    *n_tab = 0;
    if (n_words == 0 || n_words > kMaxNarrowWords) return SVO_OK;
    const uint32_t W = (uint32_t)n_words;
    if (n_words <= kWordOrderMost) {
        const int rc = build_word_order(d_words, n_words, levels, st, tab, n_tab);
        if (rc != SVO_OK || *tab) return rc;
    }
    // per level, the nodes' words and their first children within the next:
    // 8 bytes a node until the table itself can be had
    constexpr int kMost = kTableMaxParentLevel + 2;
    std::unique_ptr<Scratch[]> nodes(new Scratch[kMost + 1]), first(new Scratch[kMost + 1]);
    std::vector<uint32_t> lv_n;
    Scratch err, total;
    SVO_CUDA_TRY(err.alloc(sizeof(uint32_t), st));
    SVO_CUDA_TRY(total.alloc(sizeof(uint32_t), st));
    SVO_CUDA_TRY(cudaMemsetAsync(err.p, 0, sizeof(uint32_t), st));
    SVO_CUDA_TRY(nodes[0].alloc(sizeof(uint32_t), st));
    SVO_CUDA_TRY(cudaMemsetAsync(nodes[0].p, 0, sizeof(uint32_t), st));  // level 0: the root at word 0
    uint32_t n = 1;
    uint64_t base = 0;
    bool ok = true;
    for (int L = 0; n > 0; ++L) {
        if (L >= kMost || base + n > n_words) {
            ok = false;
            break;
        }
        const uint32_t *const at = (const uint32_t *)nodes[L].p;
        Scratch c, sc;
        SVO_CUDA_TRY(c.alloc((size_t)n * sizeof(uint32_t), st));
        SVO_CUDA_TRY(first[L].alloc((size_t)n * sizeof(uint32_t), st));
        SVO_CUDA_TRY(sc.alloc(scan_scratch_elems(n) * sizeof(uint32_t), st));
        uint32_t *const f = (uint32_t *)first[L].p;
        k_table_count<<<grid_for(n), 256, 0, st>>>(d_words, W, at, n, L, (uint32_t *)c.p, (uint32_t *)err.p);
        SVO_CUDA_TRY(cudaGetLastError());
        SVO_CUDA_TRY((exclusive_scan<uint32_t, uint32_t>((const uint32_t *)c.p, f, n, (uint32_t *)total.p,
                                                         (uint32_t *)sc.p, st)));
        uint32_t next_n = 0;
        SVO_CUDA_TRY(cudaMemcpyAsync(&next_n, total.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        SVO_CUDA_TRY(cudaStreamSynchronize(st));
        lv_n.push_back(n);
        base += n;
        if (base + next_n > n_words) {
            ok = false;
            break;
        }
        if (next_n) {
            SVO_CUDA_TRY(nodes[L + 1].alloc((size_t)next_n * sizeof(uint32_t), st));
            k_table_children<<<grid_for(n), 256, 0, st>>>(d_words, W, at, n, L, f, (uint32_t *)nodes[L + 1].p);
            SVO_CUDA_TRY(cudaGetLastError());
        }
        n = next_n;
    }
    uint32_t err_h = 0;
    SVO_CUDA_TRY(cudaMemcpyAsync(&err_h, err.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    SVO_CUDA_TRY(cudaStreamSynchronize(st));
    if (!ok || err_h) return SVO_OK;
    uint4 *t = nullptr;
    SVO_CUDA_TRY(handle_alloc((void **)&t, (size_t)base * sizeof(uint4), st));
    uint64_t at = 0;
    for (size_t L = 0; L < lv_n.size(); ++L) {
        k_table_write<<<grid_for(lv_n[L]), 256, 0, st>>>(d_words, W, (const uint32_t *)nodes[L].p, lv_n[L], (int)L,
                                                         (const uint32_t *)first[L].p, (uint32_t)(at + lv_n[L]), t + at);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            handle_free(t, (size_t)base * sizeof(uint4), st);
            return cuda_fail(e, "descriptor table");
        }
        at += lv_n[L];
    }
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        handle_free(t, (size_t)base * sizeof(uint4), st);
        return cuda_fail(e, "descriptor table");
    }
    *tab = t;
    *n_tab = base;
    return SVO_OK;
}

}  // namespace

const uint4 *octree_table(const svo_octree *oct, cudaStream_t caller) {
    if (!oct->use_table) return nullptr;
    if (oct->tab_state == 1) return oct->d_tab;
    if (oct->tab_state != 0) return nullptr;
    // Never build while the caller's stream is being captured: the checked
    // traversal runs instead, and a later uncaptured call builds the table.
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(caller, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return nullptr;
    std::lock_guard<std::mutex> lock(oct->tab_mtx);
    if (oct->tab_state == 0) {
        cudaStream_t st = nullptr;
        if (library_stream(&st) != cudaSuccess) return nullptr;
        uint4 *t = nullptr;
        uint64_t nt = 0;
        int rc = build_table(oct->d_words, oct->n_words, oct->levels, st, &t, &nt);
        if (rc != SVO_OK) {
            // A CUDA failure (device memory, most likely): keep the word
            // traversal for this handle rather than retry on every call.
            clear_error();
            cudaGetLastError();  // drop a non-sticky allocation error so later calls do not report it
            oct->tab_state = -1;
            return nullptr;
        }
        oct->d_tab = t;
        oct->n_tab = nt;
        oct->tab_state = t ? 1 : -1;
    }
    return oct->tab_state == 1 ? oct->d_tab : nullptr;
}

}  // namespace svo
