// tet_search.cuh -- the hierarchical 8 x 8 x 8 search of one tet vertex by one warp, over ring
// coefficients staged in shared memory (tet_key.cuh).
//
// Candidate filter. A level can only move the vertex to a candidate whose ring key beats the
// current key qLast, so a candidate for which any tet's key lies below qLast can be dropped. For
// qLast > 0 the condition det^2 / L^3 >= thr (thr just below qLast) is det >= sqrt(thr) L^(3/2),
// and L^(3/2) is convex in L: its tangent T(L) = 1.5 r L - 0.5 r^3 at r^2 lies below it for every
// r, so
//     g(p) = w (det(p) - sqrt(thr) T(L(p))) >= 0
// holds for every candidate that can beat qLast (w > 0 scales the tet, about 1 / r^3). det is
// affine and L an isotropic quadratic in p, so g splits into a sum of one function per axis: on
// the separable grid it is a table look-up and two additions per (candidate, tet), and the z
// additions run two at a time (f32x2) with one three-operand minimum per two tets. For thr <= 0
// (a flipped tet in the ring, whose key is its det) the condition is det(p) >= thr and the same
// form holds without the quadratic part.
// With r^2 = L at the level's centre the bound is tight: over all tets hardly a candidate survives
// that does not beat qLast (jittered cube, first five iterations: 13.5 / 4.0 / 0.1 candidates kept
// on the first level against 12.2 / 3.7 / 0.1 that beat it). The TS_CRIT tets of smallest key at
// the centre do nearly as much at a fraction of the cost; the others follow only on the coarse
// first level (whose box is too wide for the pruning below) and only while something survives.
//
// Pruning by one exact key. The smallest g of a candidate estimates how far its ring key's root
// exceeds sqrt(thr), so the candidate of the largest is judged first. When its key K1 beats qLast,
// a candidate that beats K1 needs det >= sqrt(thr1) T(L) with thr1 just below K1, hence
//     g(p) >= (sqrt(thr1) - sqrt(thr)) w T(L(p)) >= (sqrt(thr1) - sqrt(thr)) rho,
// rho the smallest w T over the box and the tets: on the second and third levels 20 to 25
// survivors shrink to one to five. What remains is judged by the full ring key.
//
// Both steps are exact: g is evaluated with its own roundings, so every tet's constant is raised by
// 2^-18 of the sum of the magnitudes that enter it, far above the few 2^-24 that det, L and g can
// be off by; an overflow makes that term infinite or NaN, and a candidate is only dropped for a
// sum that compares below the limit. Keys are the exact operations and tet order of tet_key1, and
// the winner is the largest key with the lowest linear index: positions are bit for bit those of
// the unfiltered search.
//
// Bound: issue (69 % of the slots, 2,370 to 4,975 warp instructions per vertex from the converged
// cube to the jittered start). On the 48^3 cube (20 iterations, 104 k vertices) the filter by
// fractions over six tets took 0.864 ms per iteration; this one took 0.472 ms over all tets, judging
// every survivor, and takes 0.404 ms over the critical tets with the pruning.
#pragma once
#include "tet_key.cuh"
#include "f32x2.cuh"
#include <cfloat>

namespace vsdmo {

// floats per tet: (x_i, x_i) for i = 0..7, (y_j, y_j, y_7-j, y_7-j) for j = 0..3, z in the order of
// TS_Z; 44: no bank conflicts
constexpr int TS_SLOT = 44;
constexpr int TS_TABLE = 32 * TS_SLOT;      // one round of 32 tets
// Tets looked at first (rings of up to 32) and the pruning bound below which the others follow, when
// anything survives: 6 / 8 / 10 / 12 / all tets first took 0.479 / 0.418 / 0.404 / 0.409 / 0.439 ms
// per iteration of the 48^3 cube (20 iterations), never looking at the others 0.418 (10 tets).
constexpr int TS_CRIT = 10;
constexpr float TS_RHO = 0.3f;
constexpr int TS_LIST = 512;                // survivors (16-bit candidate indices): every candidate fits
// shared memory of one warp's search besides the ring coefficients, in bytes (a multiple of 16)
constexpr int TS_WARP_BYTES = TS_TABLE * 4 + TS_LIST * 2;

// candidate offsets (N-1-2i)/(N-1): i = 0 is +extent, i = N-1 is -extent (DMOTetImplCub.h:101-103)
static __device__ __forceinline__ float grid_offset(int i) {
    switch (i) {
    case 0: return 7.0f / 7.0f;
    case 1: return 5.0f / 7.0f;
    case 2: return 3.0f / 7.0f;
    case 3: return 1.0f / 7.0f;
    case 4: return -1.0f / 7.0f;
    case 5: return -3.0f / 7.0f;
    case 6: return -5.0f / 7.0f;
    default: return -7.0f / 7.0f;
    }
}

// t[i] = (value at offset i, value at offset 7 - i) = base +- o_i P - o_i^2 Q on one axis, i = 0..3
static __device__ __forceinline__ void axis_table(float base, float P, float Q, f32x2* t) {
    const f32x2 PP = pk2(P, P);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float o = grid_offset(i);
        const float e = fmaf(-(o * o), Q, base);
        t[i] = fma2(pk2(o, -o), PP, pk2(e, e));
    }
}

// linear index of candidate (lane & 7, y place jj, z place q), i = 2 q + jj: the y places of a lane are
// j and 7 - j with j = lane >> 3, the z places 0 1 2 3 7 6 5 4
static __device__ __forceinline__ int tet_index(int lane, int i) {
    const int j = lane >> 3, q = i >> 1;
    return (lane & 7) + 8 * ((i & 1) ? 7 - j : j) + 64 * (q < 4 ? q : 11 - q);
}

// largest of the warp's 512 bounds
static __device__ __forceinline__ float top_bound(const float (&s)[16]) {
    float t = fmaxf(s[0], s[1]);
#pragma unroll
    for (int i = 2; i < 16; i += 2) t = max3(t, s[i], s[i + 1]);
    return redux_max(t);
}

// Lower bounds of the 512 candidates centre + offset * S: s[2 q + jj] of a lane is the smallest g
// of candidate tet_index(lane, 2 q + jj) over the tets looked at. sq, low: sqrt(thr) and 0,
// or 0 and thr. rho: the smallest w T over the box and those tets (0 where there is no bound).
// tab: the warp's TS_TABLE floats. Returns false when the critical tets already drop every
// candidate (most searches of a nearly converged mesh).
static __device__ __forceinline__ bool tet_quad_filter(const float4* __restrict__ co, int k, float* __restrict__ tab,
                                                       int lane, float dx, float dy, float dz, float Sx, float Sy,
                                                       float Sz, float sq, float low, float (&s)[16], float& rho) {
    constexpr unsigned FULL = 0xffffffffu;
    const float Xm = fabsf(dx) + Sx, Ym = fabsf(dy) + Sy, Zm = fabsf(dz) + Sz;
    const float R2 = fmaf(Xm, Xm, fmaf(Ym, Ym, Zm * Zm));
    const float dd = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
#pragma unroll
    for (int i = 0; i < 16; ++i) s[i] = FLT_MAX;
    rho = FLT_MAX;
    for (int t0 = 0; t0 < k; t0 += 32) {
        const int t = min(t0 + lane, k - 1);
        const float4 A = co[2 * t], B = co[2 * t + 1];
        // the tangent's point r^2 = L and its slope b = 1.5 sqrt(thr) r, all scaled by w
        const float det = fmaf(A.z, dz, fmaf(A.y, dy, fmaf(A.x, dx, A.w)));
        const float L = fmaf(3.f, dd, fmaf(B.z, dz, fmaf(B.y, dy, fmaf(B.x, dx, B.w))));
        const float r = sqrt_approx(fmaxf(L, 0.f));
        const float r3 = (r * r) * r;
        const float w = __fdividef(1.f, r3);
        const float b = 1.5f * (sq * r), a = 0.5f * (sq * r3);
        // magnitudes of all that enters g, for the rounding allowance
        const float mag = fmaf(fabsf(A.x), Xm, fmaf(fabsf(A.y), Ym, fmaf(fabsf(A.z), Zm, fabsf(A.w)))) +
                          fmaf(b, fmaf(fabsf(B.x), Xm, fmaf(fabsf(B.y), Ym, fmaf(fabsf(B.z), Zm, fmaf(3.f, R2, B.w)))),
                               a - low);
        const float g = w * (((det - low) + fmaf(-b, L, a)) + 0x1p-18f * mag);
        const float Lx = fmaf(6.f, dx, B.x), Ly = fmaf(6.f, dy, B.y), Lz = fmaf(6.f, dz, B.z);   // gradient of L
        const float wx = w * Sx, wy = w * Sy, wz = w * Sz, b3 = 3.f * b;
        const float Px = wx * fmaf(-b, Lx, A.x), Qx = b3 * (Sx * wx);
        const float Py = wy * fmaf(-b, Ly, A.y), Qy = b3 * (Sy * wy);
        const float Pz = wz * fmaf(-b, Lz, A.z), Qz = b3 * (Sz * wz);
        // a tet whose g is positive on the whole box (concave per axis: smallest at an end) drops nothing
        const float gmin = g - (((fabsf(Px) + Qx) + (fabsf(Py) + Qy)) + (fabsf(Pz) + Qz));
        const unsigned use = __ballot_sync(FULL, t0 + lane < k && !(gmin > 0.f));
        const int m = __popc(use);
        // the tets looked at first: the TS_CRIT of smallest det / r^3 (any choice is exact)
        unsigned crit = use;
        if (k <= 32) {
            if (m > TS_CRIT + 2) {
                const float v = (use >> lane) & 1u ? det * w : FLT_MAX;
                float left = v, top = 0.f;
#pragma unroll
                for (int i = 0; i < TS_CRIT; ++i) {
                    top = redux_min(left);
                    left = left > top ? left : FLT_MAX;
                }
                crit &= __ballot_sync(FULL, !(v > top));
            }
        } else if (t0) {
            __syncwarp();   // the table of the round before is no longer read
        }
        const int m1 = __popc(crit);
        const unsigned lower = (1u << lane) - 1u;
        if ((use >> lane) & 1u) {
            float* u = tab + ((crit >> lane) & 1u ? __popc(crit & lower) : m1 + __popc(use & ~crit & lower)) * TS_SLOT;
            f32x2 v[4];
            float e[8];
            axis_table(g, Px, Qx, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) upk2(v[i], e[i], e[7 - i]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *reinterpret_cast<float4*>(u + 4 * i) = make_float4(e[2 * i], e[2 * i], e[2 * i + 1], e[2 * i + 1]);
            axis_table(0.f, Py, Qy, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float y0, y1;
                upk2(v[i], y0, y1);
                *reinterpret_cast<float4*>(u + 16 + 4 * i) = make_float4(y0, y0, y1, y1);
            }
            axis_table(0.f, Pz, Qz, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) upk2(v[i], e[i], e[4 + i]);
            *reinterpret_cast<float4*>(u + 32) = make_float4(e[0], e[1], e[2], e[3]);
            *reinterpret_cast<float4*>(u + 36) = make_float4(e[4], e[5], e[6], e[7]);
            // L >= L(centre) - sum |grad L| S on the box
            const float Lmin = L - fmaf(fabsf(Lx), Sx, fmaf(fabsf(Ly), Sy, fabsf(Lz) * Sz));
            const float T = w * fmaf(1.5f * r, Lmin, -0.5f * r3);
            rho = fminf(rho, T > 0.f ? T : 0.f);
        }
        // an odd count is padded with a tet that drops nothing
        if (m & 1)
            for (int i = lane; i < 40; i += 32) tab[m * TS_SLOT + i] = i < 16 ? FLT_MAX : 0.f;
        rho = redux_min(rho);
        __syncwarp();
        const float* u = tab;
        int j = 0, end = m1;
        while (true) {
            for (; j < end; j += 2, u += 2 * TS_SLOT) {
                f32x2 xy[2][2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float* ue = u + e * TS_SLOT;
                    const f32x2 x = *reinterpret_cast<const f32x2*>(ue + 2 * (lane & 7));
                    const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(ue + 16 + 4 * (lane >> 3));
                    xy[e][0] = add2(x, y.x);
                    xy[e][1] = add2(x, y.y);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const ulonglong2 z0 = *reinterpret_cast<const ulonglong2*>(u + 32 + 4 * h);
                    const ulonglong2 z1 = *reinterpret_cast<const ulonglong2*>(u + TS_SLOT + 32 + 4 * h);
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        const f32x2 za = p ? z0.y : z0.x, zb = p ? z1.y : z1.x;
                        const int q = 4 * h + 2 * p;
#pragma unroll
                        for (int jj = 0; jj < 2; ++jj) {
                            float u0, u1, v0, v1;
                            upk2(add2(xy[0][jj], za), u0, u1);
                            upk2(add2(xy[1][jj], zb), v0, v1);
                            s[2 * q + jj] = min3(s[2 * q + jj], u0, v0);
                            s[2 * q + 2 + jj] = min3(s[2 * q + 2 + jj], u1, v1);
                        }
                    }
                }
            }
            if (j >= m) break;
            if (top_bound(s) < 0.f) return false;
            if (rho >= TS_RHO) break;
            end = m;
        }
    }
    if (!(rho < FLT_MAX)) rho = 0.f;   // no tet looked at
    return true;
}

// tet_key1 of the candidate (x, y, z) by the P lanes of an aligned group (P a power of two up to
// 32, the same on all lanes; the candidate is the group's): each lane folds every P-th tet and the
// smallest fold is the ring key. The serial fold compares fractions by cross-multiplication and
// ends on the tet whose fraction is clearly smallest; where several lanes' folds lie within
// 2^-19 of the smallest (or are not finite), the group repeats the serial fold itself, so the
// result is tet_key1's bit for bit.
static __device__ __forceinline__ float tet_group_key(const float4* __restrict__ co, int k, float x, float y, float z,
                                                      int P, int lane) {
    constexpr unsigned FULL = 0xffffffffu;
    const int sub = lane & (P - 1);
    const float tx = (3.0f * x) * x, ty = (3.0f * y) * y, tz = (3.0f * z) * z;
    float N = 0.f, D = 1.f, dm = 0.f;
    for (int t = sub; t < k; t += P) {
        const float4 c0 = co[2 * t], c1 = co[2 * t + 1];
        const float det = fmaf(c0.z, z, fmaf(c0.y, y, fmaf(c0.x, x, c0.w)));
        const float L = ((c1.w + fmaf(c1.x, x, tx)) + fmaf(c1.y, y, ty)) + fmaf(c1.z, z, tz);
        const float num = det * det, den = (L * L) * L;
        if (t == sub) { N = num; D = den; dm = det; continue; }
        if (num * D < N * den) { N = num; D = den; }
        dm = fminf(dm, det);
    }
    const float v = sub >= k ? FLT_MAX : dm < 0.f ? dm : __fdividef(N, D);
    float m = v;
    if (P == 32) m = redux_min(v);
    else for (int o = P >> 1; o; o >>= 1) m = fminf(m, __shfl_xor_sync(FULL, m, o));
    const unsigned near = __ballot_sync(FULL, sub < k && (!(v > m + fabsf(m) * 0x1p-19f) || !(D < 1e36f)));
    const unsigned mine = P == 32 ? near : (near >> (lane & ~(P - 1))) & ((1u << P) - 1u);
    const int owner = (lane & ~(P - 1)) + __ffs((int)mine) - 1;
    const float on = __shfl_sync(FULL, N, owner & 31), od = __shfl_sync(FULL, D, owner & 31);
    if (m < 0.f) return m;   // the smallest det, exact in any order
    if (__popc(mine) == 1) return on / od;
    return tet_key1(co, k, x, y, z);
}

// value just below the key q: what a candidate that beats q cannot fall under on any tet (the
// margin covers the rounding of the fraction comparisons along a ring)
static __device__ __forceinline__ float tet_below(float q) { return q - (fabsf(q) * 0x1p-14f + 1e-37f); }

// position of candidate idx; off: grid_offset(lane & 7) of every lane
static __device__ __forceinline__ float3 tet_candidate(int idx, float off, float dx, float dy, float dz, float Sx,
                                                       float Sy, float Sz) {
    constexpr unsigned FULL = 0xffffffffu;
    const float ox = __shfl_sync(FULL, off, idx & 7), oy = __shfl_sync(FULL, off, (idx >> 3) & 7);
    const float oz = __shfl_sync(FULL, off, (idx >> 6) & 7);
    return make_float3(fmaf(ox, Sx, dx), fmaf(oy, Sy, dy), fmaf(oz, Sz, dz));
}

// The plain hierarchical search (DMOTetImplCub.h:66-136) from the local origin: depth levels
// of 8 x 8 x 8 candidates, moving on strict improvement of the ring key qLast. Returns whether
// the vertex moved; (dx, dy, dz) is the new position in scaled local coordinates. scratch: the
// warp's TS_WARP_BYTES of shared memory.
//
// Up to 16 candidates are judged together by 32 / (their number, rounded up to a power of two)
// lanes each; more go one per lane, 32 at a time.
static __device__ __forceinline__ bool tet_plain_search(const float4* __restrict__ co, float* __restrict__ scratch, int k,
                                                        float sx, float sy, float sz, float grid_scale, int depth,
                                                        int lane, float qLast, float& dx, float& dy, float& dz) {
    constexpr unsigned FULL = 0xffffffffu;
    unsigned short* list = reinterpret_cast<unsigned short*>(scratch + TS_TABLE);
    const float off = grid_offset(lane & 7);   // offset i of the grid is lane i's
    dx = 0.f; dy = 0.f; dz = 0.f;
    bool moved = false;
    float ds = grid_scale;
    for (int level = 0; level < depth; ++level) {
        const float Sx = ds * sx, Sy = ds * sy, Sz = ds * sz;
        ds = ds * (2.0f / 7.0f);
        const float thr = tet_below(qLast);
        const float sq = thr > 0.f ? sqrt_approx(thr) * (1.f - 0x1p-20f) : 0.f;   // rounded down
        float s[16], rho;
        if (!tet_quad_filter(co, k, scratch, lane, dx, dy, dz, Sx, Sy, Sz, sq, thr > 0.f ? 0.f : thr, s, rho)) continue;
        // the candidate of the largest bound: the index replaces the low four bits of the bound
        float e[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) e[i] = __uint_as_float((__float_as_uint(s[i]) & ~15u) | i);
        float top = fmaxf(e[0], e[1]);
#pragma unroll
        for (int i = 2; i < 16; i += 2) top = max3(top, e[i], e[i + 1]);
        const float warp_top = redux_max(top);
        if (warp_top < 0.f) continue;   // every candidate is dropped
        float bk = -FLT_MAX;
        int bi = 1 << 30, first = -1;
        float cut = 0.f;
        if (warp_top >= 0.f) {
            const int owner = __ffs((int)__ballot_sync(FULL, top == warp_top)) - 1;
            const int i = (int)(__float_as_uint(warp_top) & 15u);
            first = owner * 16 + i;
            bi = tet_index(owner, i);
            const float3 c = tet_candidate(bi, off, dx, dy, dz, Sx, Sy, Sz);
            bk = tet_group_key(co, k, c.x, c.y, c.z, 32, lane);
            if (thr > 0.f && bk > qLast)
                cut = (sqrt_approx(tet_below(bk)) * (1.f - 0x1p-20f) - sq) * (rho * 0.999f);
            if (!(cut > 0.f)) cut = 0.f;
        }
        unsigned dead = 0;   // bit 15 - i: bound i lies below the limit
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            float u, v;
            upk2(add2(pk2(s[i], s[i + 1]), pk2(-cut, -cut)), u, v);
            dead = __funnelshift_l(__float_as_uint(u), dead, 1);
            dead = __funnelshift_l(__float_as_uint(v), dead, 1);
        }
        unsigned alive = ~dead & 0xffffu;
        if (first >> 4 == lane) alive &= ~(0x8000u >> (first & 15));
        const int cnt = __popc(alive);
        if (__any_sync(FULL, cnt)) {
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int n = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += n;
            }
            const int total = __shfl_sync(FULL, incl, 31);
            int at = incl - cnt;
            while (alive) {
                const int bit = 31 - __clz((int)alive);
                alive &= ~(1u << bit);
                list[at++] = (unsigned short)tet_index(lane, 15 - bit);
            }
            __syncwarp();
            if (total <= 16) {
                const int P = total <= 1 ? 32 : total <= 2 ? 16 : total <= 4 ? 8 : total <= 8 ? 4 : 2;
                const int idx = list[min(lane / P, total - 1)];
                const float3 c = tet_candidate(idx, off, dx, dy, dz, Sx, Sy, Sz);
                const float key = tet_group_key(co, k, c.x, c.y, c.z, P, lane);
                if (key > bk || (key == bk && idx < bi)) { bk = key; bi = idx; }
            } else {
                for (int j = lane; j - lane < total; j += 32) {
                    const int idx = list[min(j, total - 1)];
                    const float3 c = tet_candidate(idx, off, dx, dy, dz, Sx, Sy, Sz);
                    const float key = tet_key1(co, k, c.x, c.y, c.z);
                    if (key > bk || (key == bk && idx < bi)) { bk = key; bi = idx; }
                }
            }
            // largest key, lowest linear index on ties
            const float best = redux_max(bk);
            bi = (int)__reduce_min_sync(FULL, bk == best ? (unsigned)bi : 1u << 30);
            bk = best;
        }
        if (bi < 512 && qLast < bk) {
            const float3 c = tet_candidate(bi, off, dx, dy, dz, Sx, Sy, Sz);
            dx = c.x; dy = c.y; dz = c.z;
            qLast = bk;
            moved = true;
        }
        __syncwarp();   // the list and the table are rewritten by the next level
    }
    return moved;
}

}  // namespace vsdmo
