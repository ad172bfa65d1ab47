// host_tri_box.cpp — the mesh build's triangle/voxel overlap filter and exact
// test (csrc/tri_box.cuh) compiled for the host, where the float operations
// are the device's (-ffp-contract=off there is -fmad=false here).
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __forceinline__ inline
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static inline float __int_as_float(int i) {
    float f;
    std::memcpy(&f, &i, 4);
    return f;
}



#include "tri_box.cuh"

// For n triangles (9 floats each), an 8^3 brick of voxel centres (8 per axis)
// and the half voxel edge: counts[0] voxels whose box axes overlap the
// triangle's, [1] those the filter decided, [2] those it decided otherwise
// than tri_box, [3] overlaps.
extern "C" void host_filter(const float *tris, int64_t n, const float *cx, const float *cy, const float *cz, float half,
                            int64_t *counts) {
    using namespace svo;
    const float *c[3] = {cx, cy, cz};
    float o[3], cdev = 0.0f;
    for (int k = 0; k < 3; ++k) {
        o[k] = 0.5f * (c[k][0] + c[k][7]);
        for (int i = 0; i < 8; ++i) cdev = fmaxf(cdev, fabsf(c[k][i] - o[k]));
    }
    const float h[3] = {half, half, half};
    for (int64_t t = 0; t < n; ++t) {
        const float *p = tris + 9 * t;
        float F[kFltFloats] = {};
        for (int s = 0; s < 4; ++s) stage_filter(F, p, o, cdev, half, s);
        for (int v = 0; v < 512; ++v) {
            const float x = cx[v & 7], y = cy[(v >> 3) & 7], z = cz[v >> 6], at[3] = {x, y, z};
            bool box = true;
            for (int k = 0; k < 3; ++k) {
                const float a = p[k] - at[k], b = p[3 + k] - at[k], d = p[6 + k] - at[k];
                const float mn = fminf(a, fminf(b, d)), mx = fmaxf(a, fmaxf(b, d));
                if (mn > half || mx < -half) box = false;
            }
            if (!box) continue;
            const bool hit = tri_box(x, y, z, h, p);
            const float sep = filter_separation(F, x - o[0], y - o[1], z - o[2]), eps = F[kFltEps];
            const bool in = sep < -eps, out = sep > eps;
            ++counts[0];
            counts[1] += in || out;
            counts[2] += (in && !hit) || (out && hit);
            counts[3] += hit;
        }
    }
}
