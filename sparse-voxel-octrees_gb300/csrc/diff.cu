// diff.cu — differentiable leaf shading over the octree (no counterpart in
// the reference; the shading model is the viewer's shade(), Main.cpp:81-90,
// with per-leaf parameters in place of the packed leaf word).
//
// Parameters are FP32 arrays indexed by the leaf's word index (the `leaf`
// output of svo_trace): rgb[3*i..] and normal[3*i..].  For a ray with
// direction d, hitting leaf i, under light l:
//   n     = p / |p|                 (p = normal parameters; n = 0 when p = 0)
//   a     = |l.n|
//   r     = d - 2 (n.d) n           (Vec3::reflect, math/Vec3.hpp:63-71)
//   s     = max(l.r, 0)
//   rgb_k = c_k * 0.9 * a + 0.2 * s^2          (c = rgb parameters)
// Rays that hit no leaf produce 0 and no gradient.  Traversal is the discrete
// ESVO raymarch, unchanged; only the shading is differentiated:
//   dL/dc_k = g_k 0.9 a
//   dL/dn   = (0.9 sgn(l.n) sum_k g_k c_k) l - 0.8 G s [s > 0] ((n.d) l + (n.l) d),  G = sum_k g_k
//   dL/dp   = (dL/dn - n (n.dL/dn)) / |p|
// with g = dL/drgb.  Gradients are summed over rays with atomics; lanes of a
// warp that hit the same leaf are first reduced in registers (match_any +
// pointer jumping along each leaf's lanes), so one lane per distinct leaf
// issues the atomics.  Summation order across warps is not fixed, so gradients can
// differ in the last bits between runs.
#include "svo_device.cuh"
#include "svo_internal.h"

namespace svo {
namespace {

struct DiffArgs {
    const uint32_t *oct;
    const uint4 *tab;  // descriptor table (kernels instantiated with kTab)
    uint32_t n_words;
    const float *rays;
    uint32_t width, height, n_views;  // image = width x (height * n_views), view v = rows [v*height, (v+1)*height)
    uint32_t tiles_x;
    uint64_t total;
    const float *lights;  // 3 per view (device)
    const float *p_rgb, *p_n;
    uint32_t stride;  // floats from one leaf's parameters (and gradients) to the next
    uint32_t *hit_leaf;
    float *rgb;
    const float *d_rgb;
    float *g_rgb, *g_n;
    uint32_t *status;
    // fused L2 loss (svo_diff_backward_l2): dL/drgb = loss_scale (rgb - target)
    const float *target;
    float loss_scale;
    double *loss_sum;  // optional: += sum over rays and channels of (rgb - target)^2
    // optional record of the leaves that received a gradient
    uint32_t *touched;     // one bit per octree word
    uint32_t *leaf_list;   // leaves in order of first touch
    uint32_t *leaf_count;  // entries in leaf_list
    uint32_t leaf_cap;
};

__device__ __forceinline__ bool tile_pixel(const DiffArgs &a, uint64_t slot, uint32_t &idx, uint32_t &view) {
    if (slot >= a.total) return false;
    const uint32_t tile = (uint32_t)(slot >> 5), r = (uint32_t)(slot & 31);  // tile < 2^27: 32-bit division
    const uint32_t ty = tile / a.tiles_x, tx = tile - ty * a.tiles_x;
    uint32_t px = tx * 8u + (r & 7u);
    uint32_t py = ty * 4u + (r >> 3);
    if (px >= a.width || py >= a.height * a.n_views) return false;
    idx = py * a.width + px;
    view = py / a.height;
    return true;
}

struct Shading {
    float nx, ny, nz, inv_len, ln, a, nd, s;
};

struct LeafParams {
    float c[3], p[3];  // colour and (unnormalised) normal
};

// kRec: colour and normal share one 16-byte aligned record (the normal at
// floats 3..5), read as a float4 and a float2 instead of six floats.
template <bool kRec>
__device__ __forceinline__ LeafParams load_leaf(const DiffArgs &a, uint32_t leaf) {
    LeafParams l;
    const float *c = a.p_rgb + (uint64_t)a.stride * leaf;
    if constexpr (kRec) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>(c));
        const float2 r = __ldg(reinterpret_cast<const float2 *>(c + 4));
        l.c[0] = q.x; l.c[1] = q.y; l.c[2] = q.z;
        l.p[0] = q.w; l.p[1] = r.x; l.p[2] = r.y;
    } else {
        const float *p = a.p_n + (uint64_t)a.stride * leaf;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            l.c[k] = __ldg(c + k);
            l.p[k] = __ldg(p + k);
        }
    }
    return l;
}

__device__ __forceinline__ Shading shade_terms(const LeafParams &l, float dx, float dy, float dz, float lx, float ly,
                                               float lz) {
    Shading sh;
    const float px = l.p[0], py = l.p[1], pz = l.p[2];
    float len2 = px * px + py * py + pz * pz;
    sh.inv_len = len2 > 0.0f ? 1.0f / sqrtf(len2) : 0.0f;
    sh.nx = px * sh.inv_len;
    sh.ny = py * sh.inv_len;
    sh.nz = pz * sh.inv_len;
    sh.ln = lx * sh.nx + ly * sh.ny + lz * sh.nz;
    sh.a = fabsf(sh.ln);
    sh.nd = sh.nx * dx + sh.ny * dy + sh.nz * dz;
    float proj = sh.nd * 2.0f;
    float rx = dx - sh.nx * proj, ry = dy - sh.ny * proj, rz = dz - sh.nz * proj;
    sh.s = fmaxf(lx * rx + ly * ry + lz * rz, 0.0f);
    return sh;
}

// Threads per CTA of the tracing kernels (forward, and the adjoint that traces
// again).  A warp traces one 8x4 tile; the hardware starts the next CTA where
// one has finished, so no work counter is read or reset, and a small image
// has every tile in flight at once.  The persistent form before it gave a
// warp 2 (forward) or 4 (adjoint) tiles per counter access, one after another:
// a 3-view 333x251 image took 83 us forward and now takes 52, 12 views of
// 512x512 took 164 and take 145 (256^3 scenes, 30-45 dependent steps a ray).
// Whole steps with 32, 64, 128 and 256 threads: 240, 225, 222 and 224 us.
constexpr int kTraceThreads = 128;

template <bool kTab, bool kRecord, bool kRec>
__global__ void __launch_bounds__(kTraceThreads) k_diff_forward(DiffArgs a) {
    const uint64_t slot = (uint64_t)blockIdx.x * kTraceThreads + threadIdx.x;
    RayStackFor<kTab> stk;
    uint32_t idx, view;
    if (!tile_pixel(a, slot, idx, view)) return;
    const float2 *r2 = reinterpret_cast<const float2 *>(a.rays) + 3 * (uint64_t)idx;
    float2 p0 = __ldg(r2), p1 = __ldg(r2 + 1), p2 = __ldg(r2 + 2);
    RayState st;
    ray_init_any<kTab>(st, a.oct, a.tab, p0.x, p0.y, p1.x, p1.y, p2.x, p2.y);
    RayResult res;
    while (!ray_step_any<kTab, false>(st, stk, a.oct, a.tab, a.n_words, 0.0f, res)) {
    }
    if (res.status == kFault) atomicOr(a.status, 1u);
    bool hit = res.status == kLeafHit;
    if (kRecord) a.hit_leaf[idx] = hit ? res.leaf : 0xFFFFFFFFu;
    float c0 = 0.0f, c1 = 0.0f, c2 = 0.0f;
    if (hit) {
        float lx = a.lights[3 * view], ly = a.lights[3 * view + 1], lz = a.lights[3 * view + 2];
        const LeafParams l = load_leaf<kRec>(a, res.leaf);
        Shading sh = shade_terms(l, p1.y, p2.x, p2.y, lx, ly, lz);
        float spec = sh.s * sh.s * 0.2f;
        c0 = l.c[0] * 0.9f * sh.a + spec;
        c1 = l.c[1] * 0.9f * sh.a + spec;
        c2 = l.c[2] * 0.9f * sh.a + spec;
    }
    a.rgb[3 * (uint64_t)idx] = c0;
    a.rgb[3 * (uint64_t)idx + 1] = c1;
    a.rgb[3 * (uint64_t)idx + 2] = c2;
}

// Sums v[0..5] over the lanes in `peers` (the lanes holding the same key) into
// the group's lowest lane.  Pointer jumping: every lane adds the partial sum
// of the next lane of its group and then points past what it has covered, so
// after k rounds the lane of rank r holds ranks r .. r + 2^k - 1, and the
// largest group of the warp sets the number of rounds (none in a warp of
// distinct leaves, five at most).  All 32 lanes execute every shuffle.  The
// sums are those of a binary tree over the ranks.  Finding each partner with
// __fns (a software search, five per value) bound the adjoint by instruction
// issue: 178 us for 3.1 M rays (12 views of 512x512, 256^3), 47 us with this,
// of which the 0.22 GB it reads would take 32.
__device__ __forceinline__ void group_sum6(unsigned peers, float (&v)[6]) {
    const int lane = threadIdx.x & 31;
    const unsigned above = peers & (0xfffffffeu << lane);
    int next = above ? __ffs((int)above) - 1 : 32;
    while (__any_sync(0xffffffffu, next < 32)) {
        const bool take = next < 32;
        const int src = take ? next : lane;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const float o = __shfl_sync(0xffffffffu, v[k], src);
            if (take) v[k] += o;
        }
        const int nn = __shfl_sync(0xffffffffu, next, src);
        next = take ? nn : 32;
    }
}

// Records `leaf` in the touched set the first time any warp adds a gradient
// to it (called by the one lane that adds the leaf's gradient).
__device__ __forceinline__ void mark_touched(const DiffArgs &a, uint32_t leaf) {
    const uint32_t w = leaf >> 5, bit = 1u << (leaf & 31u);
    if (__ldcg(a.touched + w) & bit) return;  // already recorded (the common case after the first pass)
    if (atomicOr(a.touched + w, bit) & bit) return;
    const uint32_t pos = atomicAdd(a.leaf_count, 1u);
    if (pos < a.leaf_cap) a.leaf_list[pos] = leaf;
}

// Adds a leaf's six gradient values.  Records (kRec) take one 16-byte and one
// 8-byte vector reduction, each value added on its own as by atomicAdd.
template <bool kRec>
__device__ __forceinline__ void add_gradient(const DiffArgs &a, uint32_t leaf, const float (&v)[6]) {
    float *gr = a.g_rgb + (uint64_t)a.stride * leaf;
    if constexpr (kRec) {
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(__cvta_generic_to_global(gr)), "f"(v[0]),
                     "f"(v[1]), "f"(v[2]), "f"(v[3])
                     : "memory");
        asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(__cvta_generic_to_global(gr + 4)), "f"(v[4]),
                     "f"(v[5])
                     : "memory");
    } else {
        float *gn = a.g_n + (uint64_t)a.stride * leaf;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            atomicAdd(gr + k, v[k]);
            atomicAdd(gn + k, v[3 + k]);
        }
    }
}

// One 8x4 tile of the adjoint.  kRetrace: recompute the hit leaf by traversal
// instead of reading hit_leaf.  kFused: dL/drgb = loss_scale (rgb - target)
// from the forward pass's rgb instead of a d_rgb array; returns this lane's
// squared error.
template <bool kTab, bool kRetrace, bool kFused, bool kRec>
__device__ __forceinline__ float adjoint_tile(const DiffArgs &a, uint64_t slot, RayStackFor<kTab> &stk) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    uint32_t idx = 0, view = 0;
    const bool live = tile_pixel(a, slot, idx, view);
    uint32_t leaf = 0xFFFFFFFFu;
    float dx = 0.f, dy = 0.f, dz = 0.f;
    if (live) {
        const float2 *r2 = reinterpret_cast<const float2 *>(a.rays) + 3 * (uint64_t)idx;
        float2 p1 = __ldg(r2 + 1), p2 = __ldg(r2 + 2);
        dx = p1.y;
        dy = p2.x;
        dz = p2.y;
        if (kRetrace) {
            float2 p0 = __ldg(r2);
            RayState st;
            ray_init_any<kTab>(st, a.oct, a.tab, p0.x, p0.y, p1.x, dx, dy, dz);
            RayResult res;
            while (!ray_step_any<kTab, false>(st, stk, a.oct, a.tab, a.n_words, 0.0f, res)) {
            }
            if (res.status == kFault) atomicOr(a.status, 1u);
            if (res.status == kLeafHit) leaf = res.leaf;
        } else {
            leaf = a.hit_leaf[idx];
        }
    }
    float sq = 0.f, g0 = 0.f, g1 = 0.f, g2 = 0.f;
    if (kFused && live) {
        // every ray adds to the loss; a miss (rgb 0) contributes no gradient
        const float *c3 = a.rgb + 3 * (uint64_t)idx, *t3 = a.target + 3 * (uint64_t)idx;
        const float e0 = c3[0] - t3[0], e1 = c3[1] - t3[1], e2 = c3[2] - t3[2];
        sq = e0 * e0 + e1 * e1 + e2 * e2;
        g0 = a.loss_scale * e0;
        g1 = a.loss_scale * e1;
        g2 = a.loss_scale * e2;
    }
    const bool contrib = leaf != 0xFFFFFFFFu;
    if (!__any_sync(FULL, contrib)) return sq;  // a tile of background
    float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (contrib) {
        float lx = a.lights[3 * view], ly = a.lights[3 * view + 1], lz = a.lights[3 * view + 2];
        const LeafParams l = load_leaf<kRec>(a, leaf);
        Shading sh = shade_terms(l, dx, dy, dz, lx, ly, lz);
        if (!kFused) {
            g0 = a.d_rgb[3 * (uint64_t)idx];
            g1 = a.d_rgb[3 * (uint64_t)idx + 1];
            g2 = a.d_rgb[3 * (uint64_t)idx + 2];
        }
        v[0] = g0 * 0.9f * sh.a;
        v[1] = g1 * 0.9f * sh.a;
        v[2] = g2 * 0.9f * sh.a;
        float sgn = sh.ln > 0.0f ? 1.0f : (sh.ln < 0.0f ? -1.0f : 0.0f);
        float wl = 0.9f * sgn * (g0 * l.c[0] + g1 * l.c[1] + g2 * l.c[2]);
        float ws = sh.s > 0.0f ? -0.8f * (g0 + g1 + g2) * sh.s : 0.0f;
        // dL/dn = wl l + ws ((n.d) l + (n.l) d)
        float gnx = wl * lx + ws * (sh.nd * lx + sh.ln * dx);
        float gny = wl * ly + ws * (sh.nd * ly + sh.ln * dy);
        float gnz = wl * lz + ws * (sh.nd * lz + sh.ln * dz);
        float ndg = sh.nx * gnx + sh.ny * gny + sh.nz * gnz;
        v[3] = (gnx - sh.nx * ndg) * sh.inv_len;
        v[4] = (gny - sh.ny * ndg) * sh.inv_len;
        v[5] = (gnz - sh.nz * ndg) * sh.inv_len;
    }
    // warp aggregation by leaf: one set of atomics per distinct leaf.  Lanes
    // without a leaf are groups of their own (they would only sum zeros).
    const unsigned lanes = __ballot_sync(FULL, contrib);
    const unsigned peers = __match_any_sync(FULL, leaf) & (contrib ? lanes : 1u << lane);
    group_sum6(peers, v);
    if (contrib && lane == __ffs((int)peers) - 1) {
        add_gradient<kRec>(a, leaf, v);
        if (a.touched) mark_touched(a, leaf);
    }
    return sq;
}

// The loss is summed in groups of four tiles: a lane adds its four squared
// errors and the lanes are added by halves, in float, and the groups' sums are
// added in double.  Both adjoint kernels group alike.
constexpr int kLossTiles = 4;

__device__ __forceinline__ float lanes_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The adjoint over recorded hit leaves: short per tile and even, so the groups
// of tiles are dealt out by a fixed stride over a resident grid, with one
// atomic on the loss per warp.
template <bool kFused, bool kRec>
__global__ void __launch_bounds__(256) k_diff_backward(DiffArgs a) {
    RayStackFor<false> stk;  // unused: nothing is traced
    double loss = 0.0;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x * kLossTiles;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    for (uint64_t s0 = warp * (32 * kLossTiles); s0 < a.total; s0 += step) {  // uniform per warp
        float group = 0.0f;
#pragma unroll 1
        for (int t = 0; t < kLossTiles; ++t)
            group += adjoint_tile<false, false, kFused, kRec>(a, s0 + (uint64_t)(32 * t) + (threadIdx.x & 31), stk);
        if (kFused && a.loss_sum) loss += (double)lanes_sum(group);
    }
    if (kFused && a.loss_sum && (threadIdx.x & 31) == 0 && loss != 0.0) atomicAdd(a.loss_sum, loss);
}

// The adjoint that traces again: a tile per warp, as the forward pass, and a
// group of tiles per CTA.
template <bool kTab, bool kFused, bool kRec>
__global__ void __launch_bounds__(kTraceThreads) k_diff_retrace(DiffArgs a) {
    static_assert(kTraceThreads == 32 * kLossTiles, "a CTA's tiles are a group");
    RayStackFor<kTab> stk;
    const uint64_t slot = (uint64_t)blockIdx.x * kTraceThreads + threadIdx.x;
    const float sq = adjoint_tile<kTab, true, kFused, kRec>(a, slot, stk);
    if (kFused && a.loss_sum) {
        __shared__ float tile_sq[kTraceThreads];
        tile_sq[threadIdx.x] = sq;
        __syncthreads();
        if (threadIdx.x < 32) {
            float group = 0.0f;
#pragma unroll
            for (int t = 0; t < kLossTiles; ++t) group += tile_sq[32 * t + threadIdx.x];
            group = lanes_sum(group);
            if (threadIdx.x == 0) atomicAdd(a.loss_sum, (double)group);
        }
    }
}

int prepare(const svo_octree *oct, const float *rays, uint32_t width, uint32_t height, uint32_t n_views,
            const float *lights, const float *p_rgb, const float *p_n, uint32_t stride, DiffArgs &a) {
    if (!oct || !rays || !lights || !p_rgb || !p_n || width == 0 || height == 0 || n_views == 0)
        return set_error(SVO_ERR_INVALID, "bad arguments");
    if (stride < 3) return set_error(SVO_ERR_INVALID, "parameter stride %u below 3", stride);
    if ((uint64_t)width * height * n_views > 0xFFFFFFFFull) return set_error(SVO_ERR_LIMIT, "more than 2^32-1 rays");
    if (wide_octree(oct)) return set_error(SVO_ERR_LIMIT, "leaf shading takes octrees of up to 2^32-1 words");
    std::memset(&a, 0, sizeof(a));
    a.oct = oct->d_words;
    a.n_words = (uint32_t)oct->n_words;
    a.rays = rays;
    a.width = width;
    a.height = height;
    a.n_views = n_views;
    a.tiles_x = (width + 7) / 8;
    a.total = (uint64_t)a.tiles_x * ((height * n_views + 3) / 4) * 32;
    a.lights = lights;
    a.p_rgb = p_rgb;
    a.p_n = p_n;
    a.stride = stride;
    a.status = oct->d_status;
    return SVO_OK;
}

// Whether the parameters form records that can be read as a float4 and a
// float2: the normal three floats after the colour, every record on a 16-byte
// boundary and at least six floats long.
bool records(const float *rgb, const float *normal, uint32_t stride) {
    return normal == rgb + 3 && stride >= 6 && stride % 4 == 0 && (reinterpret_cast<uintptr_t>(rgb) & 15) == 0;
}

template <typename K>
int launch_tiles(K kern, const DiffArgs &a, cudaStream_t st) {
    const uint64_t ctas = (a.total + kTraceThreads - 1) / kTraceThreads;  // at most 2^35 slots (a 1-pixel-wide view pads 8-fold)
    kern<<<(unsigned)ctas, kTraceThreads, 0, st>>>(a);
    SVO_CUDA_TRY(cudaGetLastError());
    return SVO_OK;
}

template <typename K>
int launch_resident(K kern, const DiffArgs &a, cudaStream_t st) {
    int dev = 0, sms = 0, resident = 0;
    SVO_CUDA_TRY(cudaGetDevice(&dev));
    SVO_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    SVO_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kern, 256, 0));
    const uint64_t need = (a.total + 255) / 256, fit = (uint64_t)sms * (resident > 0 ? resident : 1);
    kern<<<(unsigned)(need < fit ? need : fit), 256, 0, st>>>(a);
    SVO_CUDA_TRY(cudaGetLastError());
    return SVO_OK;
}

template <bool kFused>
int launch_backward(const svo_octree *oct, DiffArgs &a, cudaStream_t st) {
    const bool rec = records(a.p_rgb, a.p_n, a.stride) && records(a.g_rgb, a.g_n, a.stride);
    if (a.hit_leaf)
        return rec ? launch_resident(k_diff_backward<kFused, true>, a, st)
                   : launch_resident(k_diff_backward<kFused, false>, a, st);
    a.tab = octree_table(oct, st);  // the table only serves the retrace
    if (a.tab)
        return rec ? launch_tiles(k_diff_retrace<true, kFused, true>, a, st)
                   : launch_tiles(k_diff_retrace<true, kFused, false>, a, st);
    return rec ? launch_tiles(k_diff_retrace<false, kFused, true>, a, st)
               : launch_tiles(k_diff_retrace<false, kFused, false>, a, st);
}

template <bool kTab>
int launch_forward(const DiffArgs &a, cudaStream_t st) {
    if (records(a.p_rgb, a.p_n, a.stride))
        return a.hit_leaf ? launch_tiles(k_diff_forward<kTab, true, true>, a, st)
                          : launch_tiles(k_diff_forward<kTab, false, true>, a, st);
    return a.hit_leaf ? launch_tiles(k_diff_forward<kTab, true, false>, a, st)
                      : launch_tiles(k_diff_forward<kTab, false, false>, a, st);
}

}  // namespace
}  // namespace svo

using namespace svo;

extern "C" {

int svo_diff_forward_stride(const svo_octree *oct, const float *rays, uint32_t width, uint32_t height,
                            uint32_t n_views, const float *lights, const float *leaf_rgb, const float *leaf_normal,
                            uint32_t param_stride, uint32_t *hit_leaf, float *rgb, svo_stream stream) {
    DiffArgs a;
    int rc = prepare(oct, rays, width, height, n_views, lights, leaf_rgb, leaf_normal, param_stride, a);
    if (rc) return rc;
    if (!rgb) return set_error(SVO_ERR_INVALID, "rgb output required");
    a.hit_leaf = hit_leaf;
    a.rgb = rgb;
    cudaStream_t st = (cudaStream_t)stream;
    a.tab = octree_table(oct, st);
    return a.tab ? launch_forward<true>(a, st) : launch_forward<false>(a, st);
}

int svo_diff_backward_stride(const svo_octree *oct, const float *rays, uint32_t width, uint32_t height,
                             uint32_t n_views, const float *lights, const float *leaf_rgb, const float *leaf_normal,
                             uint32_t param_stride, const uint32_t *hit_leaf, const float *d_rgb, float *grad_rgb,
                             float *grad_normal, svo_stream stream) {
    DiffArgs a;
    int rc = prepare(oct, rays, width, height, n_views, lights, leaf_rgb, leaf_normal, param_stride, a);
    if (rc) return rc;
    if (!d_rgb || !grad_rgb || !grad_normal) return set_error(SVO_ERR_INVALID, "gradient buffers required");
    a.hit_leaf = const_cast<uint32_t *>(hit_leaf);
    a.d_rgb = d_rgb;
    a.g_rgb = grad_rgb;
    a.g_n = grad_normal;
    return launch_backward<false>(oct, a, (cudaStream_t)stream);
}

int svo_diff_backward_l2_stride(const svo_octree *oct, const float *rays, uint32_t width, uint32_t height,
                                uint32_t n_views, const float *lights, const float *leaf_rgb,
                                const float *leaf_normal, uint32_t param_stride, const uint32_t *hit_leaf,
                                const float *rgb, const float *target, float loss_scale, float *grad_rgb,
                                float *grad_normal, double *loss_sum, uint32_t *touched, uint32_t *leaf_list,
                                uint32_t *leaf_count, uint64_t leaf_capacity, svo_stream stream) {
    DiffArgs a;
    int rc = prepare(oct, rays, width, height, n_views, lights, leaf_rgb, leaf_normal, param_stride, a);
    if (rc) return rc;
    if (!rgb || !target || !grad_rgb || !grad_normal)
        return set_error(SVO_ERR_INVALID, "rgb, target and gradient buffers required");
    if ((touched != nullptr) != (leaf_list != nullptr) || (touched != nullptr) != (leaf_count != nullptr))
        return set_error(SVO_ERR_INVALID, "touched, leaf_list and leaf_count go together");
    if (touched && leaf_capacity < oct->n_words)
        return set_error(SVO_ERR_INVALID, "leaf_list holds %llu entries; it needs one per octree word (%llu)",
                         (unsigned long long)leaf_capacity, (unsigned long long)oct->n_words);
    a.hit_leaf = const_cast<uint32_t *>(hit_leaf);
    a.rgb = const_cast<float *>(rgb);
    a.target = target;
    a.loss_scale = loss_scale;
    a.loss_sum = loss_sum;
    a.g_rgb = grad_rgb;
    a.g_n = grad_normal;
    a.touched = touched;
    a.leaf_list = leaf_list;
    a.leaf_count = leaf_count;
    a.leaf_cap = touched ? (uint32_t)oct->n_words : 0u;
    return launch_backward<true>(oct, a, (cudaStream_t)stream);
}

// The separate-array forms: 3 floats per leaf in each array.
int svo_diff_forward(const svo_octree *oct, const float *rays, uint32_t width, uint32_t height, uint32_t n_views,
                     const float *lights, const float *leaf_rgb, const float *leaf_normal, uint32_t *hit_leaf,
                     float *rgb, svo_stream stream) {
    return svo_diff_forward_stride(oct, rays, width, height, n_views, lights, leaf_rgb, leaf_normal, 3, hit_leaf,
                                   rgb, stream);
}

int svo_diff_backward(const svo_octree *oct, const float *rays, uint32_t width, uint32_t height, uint32_t n_views,
                      const float *lights, const float *leaf_rgb, const float *leaf_normal, const uint32_t *hit_leaf,
                      const float *d_rgb, float *grad_rgb, float *grad_normal, svo_stream stream) {
    return svo_diff_backward_stride(oct, rays, width, height, n_views, lights, leaf_rgb, leaf_normal, 3, hit_leaf,
                                    d_rgb, grad_rgb, grad_normal, stream);
}

int svo_diff_backward_l2(const svo_octree *oct, const float *rays, uint32_t width, uint32_t height,
                         uint32_t n_views, const float *lights, const float *leaf_rgb, const float *leaf_normal,
                         const uint32_t *hit_leaf, const float *rgb, const float *target, float loss_scale,
                         float *grad_rgb, float *grad_normal, double *loss_sum, uint32_t *touched,
                         uint32_t *leaf_list, uint32_t *leaf_count, uint64_t leaf_capacity, svo_stream stream) {
    return svo_diff_backward_l2_stride(oct, rays, width, height, n_views, lights, leaf_rgb, leaf_normal, 3, hit_leaf,
                                       rgb, target, loss_scale, grad_rgb, grad_normal, loss_sum, touched, leaf_list,
                                       leaf_count, leaf_capacity, stream);
}

}  // extern "C"
