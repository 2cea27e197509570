// flat_key.cuh -- ring coefficients and keys of the 2D (flat) search, shared by the general search
// (batch.cu) and the four-vertices-per-warp search (flat_search.cuh).
#pragma once
#include <cuda_runtime.h>

namespace vsdmo {

constexpr int BCO = 9;                 // coefficient floats per ring element

static __device__ __forceinline__ float bexp2(int e) { return (e >= -126 && e <= 127) ? __int_as_float((e + 127) << 23) : 0.f; }
// x 2^e when 2^e is no normal number: kept out of line (its code at every use crowds the instruction cache)
static __device__ __noinline__ float bscale_far(float x, int e) { return ldexpf(x, e); }
static __device__ __forceinline__ float bscale(float x, float p, int e) { return p != 0.f ? x * p : bscale_far(x, e); }
// the same in line, for the general search
static __device__ __forceinline__ float bscale_here(float x, float p, int e) { return p != 0.f ? x * p : ldexpf(x, e); }

template <bool COHERENT>
static __device__ __forceinline__ float4 ldpos(const float4* p) {
    if (COHERENT) return __ldcg(p);
    return *p;
}

// triangle (p, a, b): A = K0 x + K1 y + K2, L = K5 + K3 x + K4 y + 2 |p|^2
static __device__ __forceinline__ void btri_co(float ax, float ay, float bx, float by, float* K) {
    const float ux = bx - ax, uy = by - ay;
    K[0] = -uy; K[1] = ux;
    K[2] = ax * uy - ay * ux;
    K[3] = -2.0f * (ax + bx); K[4] = -2.0f * (ay + by);
    K[5] = ((ax * ax + ay * ay) + (bx * bx + by * by)) + (ux * ux + uy * uy);
}

// quad (p, a, b, c): corner cross products c1 = K0 x + K1 y + K2, c2 = K3 x + K4 y + K5,
// edge sum l = K8 + K6 x + K7 y + 2 |p|^2
static __device__ __forceinline__ void bquad_co(float ax, float ay, float bx, float by, float cx, float cy, float* K) {
    const float e1x = bx - ax, e1y = by - ay;
    const float fx = bx - cx, fy = by - cy;
    const float gx = cx - bx, gy = cy - by;
    K[0] = -e1y; K[1] = e1x; K[2] = e1y * ax - e1x * ay;
    K[3] = fy; K[4] = -fx; K[5] = cy * fx - cx * fy;
    K[6] = -2.0f * (ax + cx); K[7] = -2.0f * (ay + cy);
    K[8] = (((ax * ax + ay * ay) + (e1x * e1x + e1y * e1y)) + (gx * gx + gy * gy)) + (cx * cx + cy * cy);
}

template <int FK>
static __device__ __forceinline__ float bkey(const float* co, int k, float x, float y) {
    const float tx = (2.0f * x) * x, ty = (2.0f * y) * y;
    float N = 0.f, D = 1.f;
    if (FK == 3) {
        float amin = 0.f;
        for (int t = 0; t < k; ++t) {
            const float* c = co + BCO * t;
            const float A = fmaf(c[1], y, fmaf(c[0], x, c[2]));
            const float L = (c[5] + fmaf(c[3], x, tx)) + fmaf(c[4], y, ty);
            if (t == 0) { N = A; D = L; amin = A; continue; }
            if (A * D < N * L) { N = A; D = L; }
            amin = fminf(amin, A);
        }
        return amin < 0.f ? amin : N / D;
    } else {
        bool neg = false;
        for (int t = 0; t < k; ++t) {
            const float* c = co + BCO * t;
            const float c1 = fmaf(c[1], y, fmaf(c[0], x, c[2]));
            const float c2 = fmaf(c[4], y, fmaf(c[3], x, c[5]));
            const float l = (c[8] + fmaf(c[6], x, tx)) + fmaf(c[7], y, ty);
            neg |= (c1 < 0.f || c2 < 0.f);
            const float num = c1 + c2;
            if (t == 0) { N = num; D = l; continue; }
            if (num * D < N * l) { N = num; D = l; }
        }
        return neg ? -1.f : N / D;
    }
}

static __device__ __forceinline__ float boffset(int i, int n) { return (float)(n - 1 - 2 * i) / (float)(n - 1); }

}  // namespace vsdmo
