// tri_box.cuh — the triangle/voxel overlap test of the mesh build: tribox3's
// arithmetic (tri_box) and a cheaper filter that decides it where it is clear.
#pragma once

namespace svo {

// Separating-axis triangle/box test of Akenine-Moller ("Fast 3D
// triangle-box overlap testing", 2001) in the form third-party/tribox3.c:
// 132-206 evaluates it: the nine edge-axis tests first (projections of two
// vertices per axis, with that code's choice of which vertex is tested
// first for the min), then the box axes, then the triangle's plane.
__device__ __forceinline__ bool axis_sep(float pa, float pb, bool a_first, float rad) {
    float mn, mx;
    if (a_first) {
        if (pa < pb) { mn = pa; mx = pb; } else { mn = pb; mx = pa; }
    } else {
        if (pb < pa) { mn = pb; mx = pa; } else { mn = pa; mx = pb; }
    }
    return mn > rad || mx < -rad;
}

__device__ __forceinline__ bool plane_box(const float n[3], const float v[3], const float h[3]) {
    float vmin[3], vmax[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
        if (n[q] > 0.0f) {
            vmin[q] = -h[q] - v[q];
            vmax[q] = h[q] - v[q];
        } else {
            vmin[q] = h[q] - v[q];
            vmax[q] = -h[q] - v[q];
        }
    }
    if (n[0] * vmin[0] + n[1] * vmin[1] + n[2] * vmin[2] > 0.0f) return false;
    if (n[0] * vmax[0] + n[1] * vmax[1] + n[2] * vmax[2] >= 0.0f) return true;
    return false;
}

__device__ __forceinline__ bool tri_box(float cx, float cy, float cz, const float h[3], const float *tv) {
    const float v0[3] = {tv[0] - cx, tv[1] - cy, tv[2] - cz};
    const float v1[3] = {tv[3] - cx, tv[4] - cy, tv[5] - cz};
    const float v2[3] = {tv[6] - cx, tv[7] - cy, tv[8] - cz};
    const float e0[3] = {v1[0] - v0[0], v1[1] - v0[1], v1[2] - v0[2]};
    const float e1[3] = {v2[0] - v1[0], v2[1] - v1[1], v2[2] - v1[2]};
    const float e2[3] = {v0[0] - v2[0], v0[1] - v2[1], v0[2] - v2[2]};
    float fex, fey, fez, a, b;

    fex = fabsf(e0[0]); fey = fabsf(e0[1]); fez = fabsf(e0[2]);
    a = e0[2]; b = e0[1];
    if (axis_sep(a * v0[1] - b * v0[2], a * v2[1] - b * v2[2], true, fez * h[1] + fey * h[2])) return false;
    a = e0[2]; b = e0[0];
    if (axis_sep(-a * v0[0] + b * v0[2], -a * v2[0] + b * v2[2], true, fez * h[0] + fex * h[2])) return false;
    a = e0[1]; b = e0[0];
    if (axis_sep(a * v1[0] - b * v1[1], a * v2[0] - b * v2[1], false, fey * h[0] + fex * h[1])) return false;

    fex = fabsf(e1[0]); fey = fabsf(e1[1]); fez = fabsf(e1[2]);
    a = e1[2]; b = e1[1];
    if (axis_sep(a * v0[1] - b * v0[2], a * v2[1] - b * v2[2], true, fez * h[1] + fey * h[2])) return false;
    a = e1[2]; b = e1[0];
    if (axis_sep(-a * v0[0] + b * v0[2], -a * v2[0] + b * v2[2], true, fez * h[0] + fex * h[2])) return false;
    a = e1[1]; b = e1[0];
    if (axis_sep(a * v0[0] - b * v0[1], a * v1[0] - b * v1[1], true, fey * h[0] + fex * h[1])) return false;

    fex = fabsf(e2[0]); fey = fabsf(e2[1]); fez = fabsf(e2[2]);
    a = e2[2]; b = e2[1];
    if (axis_sep(a * v0[1] - b * v0[2], a * v1[1] - b * v1[2], true, fez * h[1] + fey * h[2])) return false;
    a = e2[2]; b = e2[0];
    if (axis_sep(-a * v0[0] + b * v0[2], -a * v1[0] + b * v1[2], true, fez * h[0] + fex * h[2])) return false;
    a = e2[1]; b = e2[0];
    if (axis_sep(a * v1[0] - b * v1[1], a * v2[0] - b * v2[1], false, fey * h[0] + fex * h[1])) return false;

    const float *vv[3] = {v0, v1, v2};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float mn = vv[0][k], mx = vv[0][k];
        if (vv[1][k] < mn) mn = vv[1][k];
        if (vv[1][k] > mx) mx = vv[1][k];
        if (vv[2][k] < mn) mn = vv[2][k];
        if (vv[2][k] > mx) mx = vv[2][k];
        if (mn > h[k] || mx < -h[k]) return false;
    }
    const float n[3] = {e0[1] * e1[2] - e0[2] * e1[1], e0[2] * e1[0] - e0[0] * e1[2], e0[0] * e1[1] - e0[1] * e1[0]};
    return plane_box(n, v0, h);
}

// What the overlap filter keeps per staged pair, in coordinates relative to
// the brick's centre: the edges (9), the middle (9) and half width (9) of the
// interval that each of the nine edge-axis projections of the voxel's centre
// must fall in, the plane's normal, offset and half width (5), the margin.
constexpr int kFltE = 0, kFltMid = 9, kFltHalf = 18, kFltPlane = 27, kFltEps = 32, kFltFloats = 36;

// One quarter of a pair's filter constants: edge s (0..2) or the plane (3).
// p: the triangle's vertices, o: the brick's centre, cdev: the largest
// distance of a staged voxel centre from o on any axis.
//
// The filter decides tri_box's edge and plane tests where they are clear: it
// evaluates the same separations in exact-arithmetic terms (e x (p - c) =
// e x p - e x c, so only e x c is left per voxel) and trusts its sign when
// the value is more than `eps` from zero.  Everything is bounded by
// G >= |p - o|, |c - o|, half (per component) and D >= |e|; with u = 2^-24
// the error of an edge test as tri_box rounds it is at most 36 u G^2 + 18 u
// G D, the filter's own 32 u G^2 + 42 u G D, and eps = 128 u G (G + D)
// exceeds their sum nearly twofold.  The plane test's errors add up to 360 u
// G^2 D + 250 u G D^2; scaled by 1 / (4 D) they stay below the same eps.  A
// triangle the bounds do not hold for (not finite, no extent) gets eps =
// infinity: nothing is decided here and every voxel takes tri_box.
__device__ __forceinline__ void stage_filter(float *F, const float *p, const float o[3], float cdev, float half,
                                             int s) {
    float q[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) q[k] = p[k] - o[k % 3];
    float G = fmaxf(cdev, half), D = 0.0f;
#pragma unroll
    for (int k = 0; k < 9; ++k) G = fmaxf(G, fabsf(q[k]));
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        D = fmaxf(D, fabsf(q[3 + k] - q[k]));
        D = fmaxf(D, fabsf(q[6 + k] - q[3 + k]));
        D = fmaxf(D, fabsf(q[k] - q[6 + k]));
    }
    D *= 1.0001f;
    if (s < 3) {
        // edge s from vertex s to the next; its interval comes from vertex s
        // and the vertex opposite (the edge's two ends project alike)
        const int i0 = 3 * s, i1 = s == 2 ? 0 : 3 * s + 3, i2 = s == 0 ? 6 : 3 * s - 3;
        float v0[3], v1[3], v2[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            v0[k] = p[i0 + k] - o[k];
            v1[k] = p[i1 + k] - o[k];
            v2[k] = p[i2 + k] - o[k];
        }
        const float e[3] = {v1[0] - v0[0], v1[1] - v0[1], v1[2] - v0[2]};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int y = (k + 1) % 3, z = (k + 2) % 3;
            const float P0 = e[z] * v0[y] - e[y] * v0[z], P2 = e[z] * v2[y] - e[y] * v2[z];
            F[kFltE + 3 * s + k] = e[k];
            F[kFltMid + 3 * s + k] = (P0 + P2) * 0.5f;
            F[kFltHalf + 3 * s + k] = fabsf(P0 - P2) * 0.5f + half * (fabsf(e[z]) + fabsf(e[y]));
        }
    } else {
        const float e0[3] = {q[3] - q[0], q[4] - q[1], q[5] - q[2]};
        const float e1[3] = {q[6] - q[3], q[7] - q[4], q[8] - q[5]};
        const float f = 0.25f / D;
        const float nx = (e0[1] * e1[2] - e0[2] * e1[1]) * f, ny = (e0[2] * e1[0] - e0[0] * e1[2]) * f,
                    nz = (e0[0] * e1[1] - e0[1] * e1[0]) * f;
        F[kFltPlane] = nx;
        F[kFltPlane + 1] = ny;
        F[kFltPlane + 2] = nz;
        F[kFltPlane + 3] = nx * q[0] + ny * q[1] + nz * q[2];
        F[kFltPlane + 4] = half * (fabsf(nx) + fabsf(ny) + fabsf(nz));
        // every comparison is false for a NaN
        const bool fine = G < 1e6f && D > 1e-12f;
        F[kFltEps] = fine ? 0x1p-17f * G * (G + D) : __int_as_float(0x7f800000);
    }
}

// The largest of the separations over the nine edge axes and the plane, at
// the voxel centre (x, y, z) relative to the brick's: above eps the voxel and
// the triangle are apart, below -eps on every one of these axes they are not.
__device__ __forceinline__ float filter_separation(const float (&f)[kFltFloats], float x, float y, float z) {
    float m = fabsf(__fmaf_rn(f[kFltPlane], x, __fmaf_rn(f[kFltPlane + 1], y, __fmaf_rn(f[kFltPlane + 2], z, -f[kFltPlane + 3])))) -
              f[kFltPlane + 4];
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        const float ex = f[3 * s], ey = f[3 * s + 1], ez = f[3 * s + 2];
        const float lx = __fmaf_rn(ez, y, __fmaf_rn(-ey, z, -f[kFltMid + 3 * s]));
        const float ly = __fmaf_rn(ex, z, __fmaf_rn(-ez, x, -f[kFltMid + 3 * s + 1]));
        const float lz = __fmaf_rn(ey, x, __fmaf_rn(-ex, y, -f[kFltMid + 3 * s + 2]));
        m = fmaxf(m, fabsf(lx) - f[kFltHalf + 3 * s]);
        m = fmaxf(m, fabsf(ly) - f[kFltHalf + 3 * s + 1]);
        m = fmaxf(m, fabsf(lz) - f[kFltHalf + 3 * s + 2]);
    }
    return m;
}

}  // namespace svo
