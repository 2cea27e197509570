// tet_key.cuh -- the tet ring key of the plain search, shared by the interior search
// (dmo_kernels.cu) and the boundary-surface passes of tet meshes (surf_kernels.cu).
//
// Relative to the vertex and scaled by an exact power of two, the determinant of tet (p, a, b, c)
// is affine in the candidate p (det = d0 - n.p) and the sum of its six squared edge lengths
// quadratic (L = C - 2 s.p + 3|p|^2); the mean ratio 12 cbrt(9) cbrt(det^2) / L is compared
// through the monotone transform det^2 / L^3 (a flipped tet keys the ring by its most negative
// det, the analogue of the reference returning the negative volume).
#pragma once
#include <cuda_runtime.h>

namespace vsdmo {

// 2^e as a float when it is a normal number, else 0. Multiplying by it is exactly ldexpf(x, e)
// (both are the correctly rounded value of x 2^e), at the cost of one multiply.
static __device__ __forceinline__ float exp2_exact(int e) { return (e >= -126 && e <= 127) ? __int_as_float((e + 127) << 23) : 0.f; }
// x 2^e when 2^e is no normal number: kept out of line (its code at every use crowds the instruction cache)
static __device__ __noinline__ float scale2_far(float x, int e) { return ldexpf(x, e); }
static __device__ __forceinline__ float scale2(float x, float p, int e) { return p != 0.f ? x * p : scale2_far(x, e); }

// coefficients of tet (p, a, b, c) in scaled local coordinates
static __device__ __forceinline__ void tet_coeffs(float ax, float ay, float az, float bx, float by, float bz,
                                           float cx, float cy, float cz, float4& K0, float4& K1) {
    float ux = bx - ax, uy = by - ay, uz = bz - az;
    float wx = cx - ax, wy = cy - ay, wz = cz - az;
    float vx = cx - bx, vy = cy - by, vz = cz - bz;
    float nx = uy * wz - uz * wy;
    float ny = uz * wx - ux * wz;
    float nz = ux * wy - uy * wx;
    float d0 = (ax * nx + ay * ny) + az * nz;
    float sx = (ax + bx) + cx, sy = (ay + by) + cy, sz = (az + bz) + cz;
    float a2 = (ax * ax + ay * ay) + az * az;
    float b2 = (bx * bx + by * by) + bz * bz;
    float c2 = (cx * cx + cy * cy) + cz * cz;
    float u2 = (ux * ux + uy * uy) + uz * uz;
    float w2 = (wx * wx + wy * wy) + wz * wz;
    float v2 = (vx * vx + vy * vy) + vz * vz;
    K0 = make_float4(-nx, -ny, -nz, d0);
    K1 = make_float4(-2.0f * sx, -2.0f * sy, -2.0f * sz, ((((a2 + b2) + c2) + u2) + w2) + v2);
}

// key of one candidate (used for the current position)
static __device__ float tet_key1(const float4* co, int k, float x, float y, float z) {
    const float tx = (3.0f * x) * x, ty = (3.0f * y) * y, tz = (3.0f * z) * z;
    float N = 0.f, D = 1.f, dm = 0.f;
    for (int t = 0; t < k; ++t) {
        const float4 c0 = co[2 * t], c1 = co[2 * t + 1];
        float detA = fmaf(c0.x, x, c0.w);
        float LA = c1.w + fmaf(c1.x, x, tx);
        float detB = fmaf(c0.y, y, detA);
        float LB = LA + fmaf(c1.y, y, ty);
        float det = fmaf(c0.z, z, detB);
        float L = LB + fmaf(c1.z, z, tz);
        float num = det * det;
        float den = (L * L) * L;
        if (t == 0) { N = num; D = den; dm = det; continue; }
        if (num * D < N * den) { N = num; D = den; }
        dm = fminf(dm, det);
    }
    return dm < 0.f ? dm : N / D;
}

// tet_key1 of two candidates, the two folds' chains side by side in one pass over the ring
static __device__ void tet_key2(const float4* co, int k, float x0, float y0, float z0, float x1, float y1, float z1, float& q0, float& q1) {
    const float tx0 = (3.0f * x0) * x0, ty0 = (3.0f * y0) * y0, tz0 = (3.0f * z0) * z0;
    const float tx1 = (3.0f * x1) * x1, ty1 = (3.0f * y1) * y1, tz1 = (3.0f * z1) * z1;
    float N0 = 0.f, D0 = 1.f, m0 = 0.f, N1 = 0.f, D1 = 1.f, m1 = 0.f;
#pragma unroll 2
    for (int t = 0; t < k; ++t) {
        const float4 c0 = co[2 * t], c1 = co[2 * t + 1];
        const float d0 = fmaf(c0.z, z0, fmaf(c0.y, y0, fmaf(c0.x, x0, c0.w))), d1 = fmaf(c0.z, z1, fmaf(c0.y, y1, fmaf(c0.x, x1, c0.w)));
        const float L0 = ((c1.w + fmaf(c1.x, x0, tx0)) + fmaf(c1.y, y0, ty0)) + fmaf(c1.z, z0, tz0);
        const float L1 = ((c1.w + fmaf(c1.x, x1, tx1)) + fmaf(c1.y, y1, ty1)) + fmaf(c1.z, z1, tz1);
        const float n0 = d0 * d0, n1 = d1 * d1, e0 = (L0 * L0) * L0, e1 = (L1 * L1) * L1;
        if (t == 0 || n0 * D0 < N0 * e0) { N0 = n0; D0 = e0; }
        if (t == 0 || n1 * D1 < N1 * e1) { N1 = n1; D1 = e1; }
        m0 = t == 0 ? d0 : fminf(m0, d0);
        m1 = t == 0 ? d1 : fminf(m1, d1);
    }
    q0 = m0 < 0.f ? m0 : N0 / D0;
    q1 = m1 < 0.f ? m1 : N1 / D1;
}

// tet_key1 at the local origin (the vertex itself): det = d0 and L = C exactly there (every term
// that carries the candidate is a product with +-0 added to them), so the same fold runs on the
// constant coefficients alone and returns the same key
static __device__ float tet_key_origin(const float4* co, int k) {
    float N = 0.f, D = 1.f, dm = 0.f;
    for (int t = 0; t < k; ++t) {
        const float det = co[2 * t].w, L = co[2 * t + 1].w;
        const float num = det * det;
        const float den = (L * L) * L;
        if (t == 0) { N = num; D = den; dm = det; continue; }
        if (num * D < N * den) { N = num; D = den; }
        dm = fminf(dm, det);
    }
    return dm < 0.f ? dm : N / D;
}

}  // namespace vsdmo
