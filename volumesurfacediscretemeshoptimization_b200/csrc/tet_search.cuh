// tet_search.cuh -- the hierarchical 8 x 8 x 8 search of one tet vertex by one warp, over ring
// coefficients staged in shared memory (tet_key.cuh): the exact candidate filter of quad_filter.cuh
// over the tets, then full ring keys for what it keeps. Keys are the exact operations and tet order of
// tet_key1 and the winner is the largest key with the lowest linear index, so positions are bit for
// bit those of the unfiltered search. A flipped tet's key is its det, so a ring that holds one (key
// <= 0) takes the filter's linear form.
//
// The filter's bound is tight: over all tets hardly a candidate survives that does not beat the
// current key (jittered cube, first five iterations: 13.5 / 4.0 / 0.1 candidates kept on the first
// level against 12.2 / 3.7 / 0.1 that beat it). The critical tets do nearly as much at a fraction of
// the cost; the others follow only on the coarse first level (whose box is too wide for the pruning
// by the best key) and only while something survives. On the second and third levels 20 to 25
// survivors shrink to one to five after the first exact key.
//
// Bound: issue (69 % of the slots, 2,370 to 4,975 warp instructions per vertex from the converged
// cube to the jittered start). On the 48^3 cube (20 iterations, 104 k vertices) the filter by
// fractions over six tets took 0.864 ms per iteration; this one took 0.472 ms over all tets, judging
// every survivor, and took 0.404 ms over the critical tets with the pruning (0.400 with chained classes); it takes
// 0.412 ms with the check for rings that the filter does not hold for and the search that they take instead.
#pragma once
#include "tet_key.cuh"
#include "quad_filter.cuh"

namespace vsdmo {

// Ring keys are a minimum over the tets, in whatever order they are folded, only while every L is positive
// and its cube and the products of the fold are normal numbers: at a candidate beside a tet's collapsed base
// the rounding of L decides, and NaN positions make the fold depend on the order. Rings with a tet whose L is
// not bounded above the limit (in units of the ring's extent; edges of a quarter of a percent) on the search box are searched
// without the filter.
static __device__ __forceinline__ float tet_odd_limit(float grid_scale) { return 0x1p-16f * fmaxf(1.f, grid_scale * grid_scale); }
// L of a tet where its gradient vanishes: below L everywhere; NaN when a corner is
static __device__ __forceinline__ float tet_least(float4 K1) {
    return fmaf(-1.f / 12.f, fmaf(K1.x, K1.x, fmaf(K1.y, K1.y, K1.z * K1.z)), K1.w);
}
// the same bound from the box's distances to the corners a, b, c (the levels' half-extents sum to at most 1.4 grid_scale)
static __device__ __noinline__ bool tet_odd(float3 a, float3 b, float3 c, float grid_scale, float sx, float sy, float sz) {
    const float X = (1.5f * grid_scale) * sx, Y = (1.5f * grid_scale) * sy, Z = (1.5f * grid_scale) * sz;
    const float3 p[3] = { a, b, c };
    float d = 0.f, sum = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float x = fmaxf(fabsf(p[i].x) - X, 0.f), y = fmaxf(fabsf(p[i].y) - Y, 0.f), z = fmaxf(fabsf(p[i].z) - Z, 0.f);
        d += (x * x + y * y) + z * z;
        sum += (p[i].x + p[i].y) + p[i].z;
    }
    return sum != sum || !(d > tet_odd_limit(grid_scale));
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

// the ring's tets as filter items
struct TetItems {
    const float4* co;
    int k;
    __device__ __forceinline__ int items() const { return k; }
    __device__ __forceinline__ bool groups() const { return true; }
    __device__ __forceinline__ void load(int t, float4& A, float4& B, float& alpha) const {
        A = co[2 * t];
        B = co[2 * t + 1];
        alpha = 3.f;
    }
    __device__ __forceinline__ float group_key(float x, float y, float z, int P, int lane) const {
        return tet_group_key(co, k, x, y, z, P, lane);
    }
    __device__ __forceinline__ float key(float x, float y, float z) const { return tet_key1(co, k, x, y, z); }
};

// The plain hierarchical search (DMOTetImplCub.h:66-136) from the local origin: depth levels
// of 8 x 8 x 8 candidates, moving on strict improvement of the ring key qLast. Returns whether
// the vertex moved; (dx, dy, dz) is the new position in scaled local coordinates. scratch: the
// warp's TS_WARP_BYTES of shared memory.
static __device__ __forceinline__ bool tet_plain_search(const float4* __restrict__ co, float* __restrict__ scratch, int k,
                                                        float sx, float sy, float sz, float grid_scale, int depth,
                                                        int lane, float qLast, float& dx, float& dy, float& dz) {
    const TetItems ring{co, k};
    unsigned short* list = reinterpret_cast<unsigned short*>(scratch + TS_TABLE);
    const float off = grid_offset(lane & 7);   // offset i of the grid is lane i's
    dx = 0.f; dy = 0.f; dz = 0.f;
    bool moved = false;
    float ds = grid_scale;
    for (int level = 0; level < depth; ++level) {
        const float thr = key_below(qLast);
        const float sq = thr > 0.f ? sqrt_approx(thr) * (1.f - 0x1p-20f) : 0.f;   // rounded down
        const QuadLevel lv{dx, dy, dz, ds * sx, ds * sy, ds * sz, sq, thr > 0.f ? 0.f : thr, 0.f, false};
        ds = ds * (2.0f / 7.0f);
        float s[16], rho, above;
        int m;
        if (k <= 32) {
            if (!quad_filter<TetItems, false, true>(ring, lv, scratch, lane, s, rho, above, nullptr, m)) continue;
        } else {
            quad_filter<TetItems, false, false>(ring, lv, scratch, lane, s, rho, above, nullptr, m);
        }
        int bi, place;
        const float top = top_candidate(s, bi, place);
        if (top < 0.f) continue;   // every candidate is dropped
        float bk = -FLT_MAX, cut = 0.f;
        if (top >= 0.f) {
            const float3 c = grid_candidate(bi, off, lv);
            bk = ring.group_key(c.x, c.y, c.z, 32, lane);
            if (thr > 0.f && bk > qLast) cut = (sqrt_approx(key_below(bk)) * (1.f - 0x1p-20f) - sq) * (rho * 0.999f);
            if (!(cut > 0.f)) cut = 0.f;
        } else {   // only NaN bounds
            place = -1;
            bi = 1 << 30;
        }
        unsigned alive = at_least(s, cut);
        if (place >> 4 == lane) alive &= ~(0x8000u >> (place & 15));
        judge(ring, lv, alive, off, list, lane, bk, bi);
        if (bi < 512 && qLast < bk) {
            const float3 c = grid_candidate(bi, off, lv);
            dx = c.x; dy = c.y; dz = c.z;
            qLast = bk;
            moved = true;
        }
    }
    return moved;
}

// The same search of a ring whose keys depend on the order of its tets (odd): every candidate by tet_key1. NaN keys never win.
static __device__ __forceinline__ bool tet_full_search(const float4* __restrict__ co, int k, float sx, float sy, float sz,
                                                       float grid_scale, int depth, int lane, float& dx, float& dy, float& dz) {
    constexpr unsigned FULL = 0xffffffffu;
    const float off = grid_offset(lane & 7);
    dx = 0.f; dy = 0.f; dz = 0.f;
    bool moved = false;
    float ds = grid_scale, qLast = tet_key1(co, k, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int level = 0; level < depth; ++level) {
        const QuadLevel lv{dx, dy, dz, ds * sx, ds * sy, ds * sz, 0.f, 0.f, 0.f, false};
        ds = ds * (2.0f / 7.0f);
        float bk = -FLT_MAX;
        int bi = 1 << 30;
#pragma unroll 1
        for (int i = lane; i < 512; i += 32) {
            const float3 c = grid_candidate(i, off, lv);
            const float key = tet_key1(co, k, c.x, c.y, c.z);
            if (key > bk) { bk = key; bi = i; }
        }
        const float best = redux_max(bk);
        bi = (int)__reduce_min_sync(FULL, bk == best ? (unsigned)bi : 1u << 30);
        if (bi < 512 && qLast < best) {
            const float3 c = grid_candidate(bi, off, lv);
            dx = c.x; dy = c.y; dz = c.z;
            qLast = best;
            moved = true;
        }
    }
    return moved;
}

static __device__ __forceinline__ bool tet_search(const float4* __restrict__ co, float* __restrict__ scratch, int k, bool odd,
                                                  float sx, float sy, float sz, float grid_scale, int depth, int lane, float& dx,
                                                  float& dy, float& dz) {
    if (odd) return tet_full_search(co, k, sx, sy, sz, grid_scale, depth, lane, dx, dy, dz);
    const float qLast = tet_group_key(co, k, 0.f, 0.f, 0.f, 32, lane);
    return tet_plain_search(co, scratch, k, sx, sy, sz, grid_scale, depth, lane, qLast, dx, dy, dz);
}

}  // namespace vsdmo
