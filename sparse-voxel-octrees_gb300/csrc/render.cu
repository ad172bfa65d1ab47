// render.cu — the viewer's frame on the GPU: renderBatch + renderTile
// (Main.cpp:92-202) with the beam prepass, headless.
//
// The frame is cut into n_strips horizontal strips as Main.cpp:349-361 cuts
// it over its threads; each strip has its own corner grid (a corner every 8
// pixels, one tile row and column past the strip) and its own running
// dx/dy sums, so pixel values depend on that layout, which is a parameter.
//   1. k_corners: one thread per corner, 8x4 corners of a strip per warp; the
//      level-of-detail raymarch from the camera with coarseScale = 16 /
//      (planeDist * H) gives t or a miss depth of 1e10 (Main.cpp:166-185).
//   2. k_tiles: one warp per 8x4 half of an 8x8 tile.  A tile whose four
//      corner depths are all misses stays 0 (the strip's memset, :160);
//      otherwise each pixel rebuilds its direction from the same running
//      sums as renderTile (dx = -1 + x0*scale, then += scale per pixel),
//      normalises it with invSqrt, traces from pos + dir*max(minT - 0.03, 0)
//      (:187-198) and packs shade() as RGBA8 with the reference's
//      double-precision scale (:116-128).  With pixel_stride > 1 (the
//      viewer's half-size mode) a pixel takes the colour of its stride
//      corner (k_tiles_coarse).
#include <algorithm>
#include <cmath>

#include "chain.cuh"
#include "svo_device.cuh"
#include "svo_internal.h"

namespace svo {
namespace {

constexpr int kTile = 8;
constexpr float kTreeMiss = 1e10f;
// 1280x720 over a 1024^3 terrain: 156 us with 256-thread CTAs and the sums'
// own launch; 143, 142 and 146 with 64, 128 and 256 threads without it.
constexpr int kFrameThreads = 128;

struct FrameArgs {
    const uint32_t *oct;
    const uint4 *tab;  // descriptor table (kernels instantiated with kTab)
    uint32_t n_words;
    float a[9];
    float pos[3];
    float light[3];
    float zx, zy, zz, scale, tile_scale, aspect, coarse;
    int W, H, strip_rows, n_strips, tiles_x, tiles_y_max, pixel_stride;
    int strip_tiles;    // tiles of a whole strip (all but the last that holds rows)
    float *depth;       // n_strips x tiles_y_max x tiles_x
    uint32_t *out;
    uint32_t *status;
};

__device__ __forceinline__ void view_dir(const FrameArgs &f, float dx, float dy, float &x, float &y, float &z) {
    x = dx * f.a[0] + dy * f.a[1] + f.zx;
    y = dx * f.a[3] + dy * f.a[4] + f.zy;
    z = dx * f.a[6] + dy * f.a[7] + f.zz;
    float s = inv_sqrt(x * x + y * y + z * z);
    x *= s;
    y *= s;
    z *= s;
}

__device__ __forceinline__ int strip_rows_of(const FrameArgs &f, int s, int &y0) {
    y0 = s * f.strip_rows;
    int y1 = min((s + 1) * f.strip_rows, f.H);
    return y1 - y0;
}

// The corner loop's running sums (Main.cpp:166-168) are formed by every thread
// for itself: dx from -1 + x0*scale (x0 = 0), dy per strip from AspectRatio -
// y0*scale, stepping by tileScale.  A launch that left them in an array took
// longer than the additions (4 us and a dependent launch, against 160 float
// additions for 1280 pixels).
template <bool kTab>
__global__ void __launch_bounds__(kFrameThreads) k_corners(FrameArgs f, int warps_x) {
    chain_next();
    const int lane = threadIdx.x & 31, w = (blockIdx.x * kFrameThreads + threadIdx.x) >> 5, s = blockIdx.y;
    const int tx = (w % warps_x) * 8 + (lane & 7), ty = (w / warps_x) * 4 + (lane >> 3);
    if (tx >= f.tiles_x) return;
    int y0;
    const int rows = strip_rows_of(f, s, y0);
    const int tiles_y = (rows - 1) / kTile + 2;  // Main.cpp:360 (C division)
    if (ty >= tiles_y) return;
    float dx = -1.0f + 0.0f * f.scale;
    for (int i = 0; i < tx; ++i) dx += f.tile_scale;
    float dy = f.aspect - (float)(s * f.strip_rows) * f.scale;
    for (int i = 0; i < ty; ++i) dy -= f.tile_scale;
    float x, y, z;
    view_dir(f, dx, dy, x, y, z);
    RayResult r = trace_ray<kTab>(f.oct, f.tab, f.n_words, f.pos[0], f.pos[1], f.pos[2], x, y, z, f.coarse);
    if (r.status == kFault) atomicOr(f.status, 1u);
    f.depth[((size_t)s * f.tiles_y_max + ty) * f.tiles_x + tx] = (r.status == kLeafHit || r.status == kLodHit) ? r.t : kTreeMiss;
}

// The strip and place of a tile, and the least of its corners' depths.  Whole
// strips come first, so a tile's strip is a division; a tile past the last
// rows has no pixel (ty0 is then at or past y1).
struct TilePlace {
    int tx0, ty0, y1;
    float min_t;
};

__device__ __forceinline__ TilePlace tile_place(const FrameArgs &f, int tile) {
    const int s = min(tile / f.strip_tiles, f.n_strips - 1), k = tile - s * f.strip_tiles;
    const int c = k % (f.tiles_x - 1), r = k / (f.tiles_x - 1);
    TilePlace t;
    int y0;
    t.y1 = strip_rows_of(f, s, y0);
    t.y1 += y0;
    t.tx0 = c * kTile;
    t.ty0 = r * kTile + y0;
    t.min_t = kTreeMiss;
    if (t.ty0 < t.y1) {
        const float *d = f.depth + (size_t)s * f.tiles_y_max * f.tiles_x;
        const int idx = (r + 1) * f.tiles_x + (c + 1);
        t.min_t = smin(smin(d[idx], d[idx - 1]), smin(d[idx - f.tiles_x], d[idx - f.tiles_x - 1]));
    }
    return t;
}

// The colour of pixel (cx, cy) of a tile some corner of which hit.
template <bool kTab>
__device__ __forceinline__ uint32_t pixel_color(const FrameArgs &f, const TilePlace &t, int cx, int cy) {
    float dx = -1.0f + (float)t.tx0 * f.scale;
    for (int i = t.tx0; i < cx; ++i) dx += f.scale;
    float dy = f.aspect - (float)t.ty0 * f.scale;
    for (int i = t.ty0; i < cy; ++i) dy -= f.scale;
    float x, y, z;
    view_dir(f, dx, dy, x, y, z);
    const float t0 = smax(t.min_t - 0.03f, 0.0f);
    RayResult res = trace_ray<kTab>(f.oct, f.tab, f.n_words, f.pos[0] + x * t0, f.pos[1] + y * t0, f.pos[2] + z * t0,
                                    x, y, z, 0.0f);
    if (res.status == kFault) atomicOr(f.status, 1u);
    float col = 0.0f;
    if (res.status == kLeafHit) col = shade_grey(res.word, x, y, z, f.light[0], f.light[1], f.light[2]);
    return pack_rgba8(col);
}

// A warp per 8x4 half tile.
template <bool kTab>
__global__ void __launch_bounds__(kFrameThreads) k_tiles(FrameArgs f, int total_tiles) {
    chain_begin();
    const int lane = threadIdx.x & 31;
    const int w = (int)(((uint64_t)blockIdx.x * kFrameThreads + threadIdx.x) >> 5);
    if ((w >> 1) >= total_tiles) return;
    const TilePlace t = tile_place(f, w >> 1);
    const int px = t.tx0 + (lane & 7), py = t.ty0 + (w & 1) * 4 + (lane >> 3);
    if (px >= f.W || py >= t.y1) return;
    f.out[(size_t)py * f.W + px] = t.min_t != kTreeMiss ? pixel_color<kTab>(f, t, px, py) : 0u;
}

// pixel_stride > 1 (the viewer's half-size mode uses 3): a tile has only
// edge^2 colours, edge = ceil(8 / stride).  A warp takes as many tiles as its
// lanes hold colours for, traces those, and writes the tiles' pixels from
// them: 1280x720 at stride 3 over a 1024^3 terrain 121 us with every pixel
// traced, 90 with this.
template <bool kTab>
__global__ void __launch_bounds__(kFrameThreads) k_tiles_coarse(FrameArgs f, int total_tiles, int edge, int per_warp) {
    chain_begin();
    const int lane = threadIdx.x & 31;
    const int w = (int)(((uint64_t)blockIdx.x * kFrameThreads + threadIdx.x) >> 5);
    const int first = w * per_warp, n = min(per_warp, total_tiles - first);
    if (n <= 0) return;  // uniform per warp
    const int own = lane / (edge * edge), j = lane - own * edge * edge;
    uint32_t color = 0;
    if (own < n) {
        const TilePlace t = tile_place(f, first + own);
        const int cx = t.tx0 + (j % edge) * f.pixel_stride, cy = t.ty0 + (j / edge) * f.pixel_stride;
        if (cx < f.W && cy < t.y1 && t.min_t != kTreeMiss) color = pixel_color<kTab>(f, t, cx, cy);
    }
    __syncwarp();
    for (int g = 0; g < n; ++g) {
        const TilePlace t = tile_place(f, first + g);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int lx = lane & 7, ly = half * 4 + (lane >> 3);
            const uint32_t c = __shfl_sync(0xffffffffu, color,
                                           g * edge * edge + (ly / f.pixel_stride) * edge + lx / f.pixel_stride);
            if (t.tx0 + lx < f.W && t.ty0 + ly < t.y1) f.out[(size_t)(t.ty0 + ly) * f.W + t.tx0 + lx] = c;
        }
    }
}

}  // namespace
}  // namespace svo

using namespace svo;

extern "C" int svo_render_frame(const svo_octree *oct, const float rot[9], const float pos[3], uint32_t width,
                                uint32_t height, uint32_t n_strips, uint32_t pixel_stride, uint32_t *rgba,
                                svo_stream stream) {
    clear_error();
    if (!oct || !rot || !pos || !rgba) return set_error(SVO_ERR_INVALID, "null argument");
    if (width < 1 || height < 1 || width > 32768 || height > 32768)
        return set_error(SVO_ERR_INVALID, "frame size %ux%u outside [1, 32768]", width, height);
    if (n_strips < 1 || n_strips > height) return set_error(SVO_ERR_INVALID, "n_strips must lie in [1, height]");
    if (pixel_stride < 1 || pixel_stride > kTile) return set_error(SVO_ERR_INVALID, "pixel_stride must lie in [1, 8]");
    if (wide_octree(oct)) return set_error(SVO_ERR_LIMIT, "frame rendering takes octrees of up to 2^32-1 words");
    cudaStream_t st = (cudaStream_t)stream;
    FrameArgs f;
    f.oct = oct->d_words;
    f.tab = octree_table(oct, (cudaStream_t)stream);
    f.n_words = (uint32_t)oct->n_words;
    for (int i = 0; i < 9; ++i) f.a[i] = rot[i];
    for (int i = 0; i < 3; ++i) f.pos[i] = pos[i];
    const int W = (int)width, H = (int)height, S = (int)n_strips;
    // Main.cpp:150-158, 62
    const float plane_dist = 1.0f / std::tan(3.14159265358979323846f / 6.0f);
    f.scale = 2.0f / (float)W;
    const float tile_scale = (float)kTile * f.scale;
    f.aspect = (float)H / (float)W;
    f.zx = plane_dist * rot[2];
    f.zy = plane_dist * rot[5];
    f.zz = plane_dist * rot[8];
    f.coarse = 2.0f * (float)kTile / (plane_dist * (float)H);
    float l[3] = {rot[0] * -1.0f + rot[1] * 1.0f + rot[2] * -1.0f + 0.0f,
                  rot[3] * -1.0f + rot[4] * 1.0f + rot[5] * -1.0f + 0.0f,
                  rot[6] * -1.0f + rot[7] * 1.0f + rot[8] * -1.0f + 0.0f};
    const float inv = 1.0f / std::sqrt(l[0] * l[0] + l[1] * l[1] + l[2] * l[2]);
    for (int i = 0; i < 3; ++i) f.light[i] = l[i] * inv;
    f.W = W;
    f.H = H;
    f.n_strips = S;
    f.strip_rows = (H - 1) / S + 1;  // Main.cpp:349
    f.tiles_x = (W - 1) / kTile + 2;
    f.tiles_y_max = (f.strip_rows - 1) / kTile + 2;
    f.pixel_stride = (int)pixel_stride;
    f.tile_scale = tile_scale;
    f.strip_tiles = ((f.strip_rows - 1) / kTile + 1) * (f.tiles_x - 1);
    int total_tiles = 0;  // whole strips, then at most one with fewer rows
    for (int s = 0; s < S && s * f.strip_rows < H; ++s)
        total_tiles += ((std::min((s + 1) * f.strip_rows, H) - s * f.strip_rows - 1) / kTile + 1) * (f.tiles_x - 1);
    void *scratch = nullptr;
    const size_t n_depth = (size_t)S * f.tiles_y_max * f.tiles_x;
    SVO_CUDA_TRY(scratch_alloc(&scratch, n_depth * sizeof(float), st));
    f.depth = (float *)scratch;
    f.out = rgba;
    f.status = oct->d_status;
    const int warps_x = (f.tiles_x + 7) / 8, warps = warps_x * ((f.tiles_y_max + 3) / 4);
    const dim3 g1((unsigned)((warps * 32 + kFrameThreads - 1) / kFrameThreads), (unsigned)S);
    if (f.tab)
        k_corners<true><<<g1, kFrameThreads, 0, st>>>(f, warps_x);
    else
        k_corners<false><<<g1, kFrameThreads, 0, st>>>(f, warps_x);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && total_tiles > 0) {
        const int edge = (kTile + f.pixel_stride - 1) / f.pixel_stride, per_warp = 32 / std::min(32, edge * edge);
        const uint64_t warps2 = f.pixel_stride == 1 ? 2ull * total_tiles : ((uint64_t)total_tiles + per_warp - 1) / per_warp;
        const unsigned g2 = (unsigned)((warps2 * 32 + kFrameThreads - 1) / kFrameThreads);
        if (f.pixel_stride > 1)
            e = launch_chained(f.tab ? k_tiles_coarse<true> : k_tiles_coarse<false>, g2, kFrameThreads, st, f, total_tiles,
                               edge, per_warp);
        else
            e = launch_chained(f.tab ? k_tiles<true> : k_tiles<false>, g2, kFrameThreads, st, f, total_tiles);
    }
    cudaFreeAsync(scratch, st);
    if (e != cudaSuccess) return cuda_fail(e, "svo_render_frame");
    return SVO_OK;
}
