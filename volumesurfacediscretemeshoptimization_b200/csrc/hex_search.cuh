// hex_search.cuh -- the hierarchical 8 x 8 x 8 search of one hex vertex by one warp, over the halfhex
// coefficients of hex_key.cuh in shared memory: the exact candidate filter of quad_filter.cuh over
// the five sub-tets per halfhex that touch the candidate, then full ring keys (the operations and
// order of hex_key1) for what it keeps.
//
// The reference's block of 128 threads carries each thread's maximum across the levels
// (DMOHexImplCub.h:66-136). A carried maximum is at most the current key, and a level moves the
// vertex only on a strictly larger one, so the rule is an arg-max over the candidates above the
// current key with the lowest linear index on ties, and the final comparison against the start holds
// exactly when a level moved the vertex.
//
// The other four sub-tets per halfhex do not depend on the candidate; their smallest fraction is the
// constant key Q (the fold over the constants in ring order). A candidate whose touching sub-tets all
// lie clearly above Q has exactly the key Q (the fold ends on the constants whatever the others are),
// so where Q bounds the box it needs no key: it does not move a vertex whose current key is >= Q, and
// otherwise all such candidates tie and the lowest index among them is taken from the bounds.
// Candidates within rounding of Q on some sub-tet are judged. A halfhex whose constant part is
// degenerate makes every key zero and the vertex stays.
//
// The grid spans the per-axis minimum ring distance, so boxes are small (and shrink as the lattice
// straightens): an upper bound U of the ring keys on the box is close to the current key, and keys are
// folded over the few sub-tets that can lie below U (one to four, of 72).
#pragma once
#include "hex_key.cuh"
#include "quad_filter.cuh"

namespace vsdmo {

// item i: halfhex i / 6, its constant part (i % 6 == 0) or touching sub-tet i % 6 - 1, the order of hex_key1
struct HexItems {
    const float* co;
    int k;
    float es, ea;
    const unsigned short* subset;   // the level's items that decide its keys, and their number
    int m;
    __device__ __forceinline__ int items() const { return 6 * k; }
    __device__ __forceinline__ bool groups() const { return m > 8; }
    __device__ __forceinline__ float min_det() const { return es; }
    __device__ __forceinline__ float min_len() const { return ea; }
    __device__ __forceinline__ bool constant(int i) const { return i % 6 == 0; }
    __device__ __forceinline__ bool keep(int i, float sq2) const {
        const float* c = co + HEX_CO * (i / 6);
        return !(c[0] > (sq2 * sq2) * c[1]);
    }
    __device__ __forceinline__ void load(int i, float4& A, float4& B, float& alpha) const {
        const int h = i / 6, j = i - 6 * h - 1;
        if (j < 0) {   // positive everywhere: drops nothing
            A = make_float4(0.f, 0.f, 0.f, 1e30f);
            B = make_float4(0.f, 0.f, 0.f, 1.f);
            alpha = 0.f;
            return;
        }
        const float* q = co + HEX_CO * h + 3 + 8 * j;
        A = make_float4(q[0], q[1], q[2], q[3]);
        B = make_float4(q[4], q[5], q[6], q[7]);
        alpha = (j == 1 || j == 4) ? 3.f : 1.f;
    }
    // hex_key1 folded over the level's subset
    __device__ __forceinline__ float key(float x, float y, float z) const {
        const float t1x = x * x, t1y = y * y, t1z = z * z;
        const float t3x = (3.f * x) * x, t3y = (3.f * y) * y, t3z = (3.f * z) * z;
        float N = 0.f, D = 1.f;
        bool first = true, zero = false;
        for (int e = 0; e < m; ++e) {
            const int i = subset[e], h = i / 6, j = i - 6 * h - 1;
            const float* c = co + HEX_CO * h;
            if (j < 0) {
                if (first) { N = c[0]; D = c[1]; first = false; }
                else if (c[0] * D < N * c[1]) { N = c[0]; D = c[1]; }
                continue;
            }
            const float* q = c + 3 + 8 * j;
            const bool a3 = (j == 1 || j == 4);
            const float s = fmaf(q[0], x, fmaf(q[1], y, fmaf(q[2], z, q[3])));
            const float A = ((q[7] + fmaf(q[6], z, a3 ? t3z : t1z)) + fmaf(q[5], y, a3 ? t3y : t1y)) + fmaf(q[4], x, a3 ? t3x : t1x);
            hex_frac(s, A, es, ea, N, D, first, zero);
        }
        return zero ? 0.f : N / D;
    }
    // hex_key1 by the P lanes of an aligned group, like tet_group_key: each lane folds every P-th of
    // the 6 k fractions (a halfhex's constant part and five sub-tets); lanes within 2^-19 of the
    // smallest fold repeat the serial one
    __device__ __forceinline__ float group_key(float x, float y, float z, int P, int lane) const {
        constexpr unsigned FULL = 0xffffffffu;
        const int sub = lane & (P - 1);
        const float t1x = x * x, t1y = y * y, t1z = z * z;
        const float t3x = (3.f * x) * x, t3y = (3.f * y) * y, t3z = (3.f * z) * z;
        float N = 0.f, D = 1.f;
        bool first = true, zero = false;
        for (int i = sub; i < 6 * k; i += P) {
            const int h = i / 6, j = i - 6 * h;
            const float* c = co + HEX_CO * h;
            if (j == 0) {
                if (c[2] != 0.f) zero = true;
                else if (first) { N = c[0]; D = c[1]; first = false; }
                else if (c[0] * D < N * c[1]) { N = c[0]; D = c[1]; }
            } else {
                const float* q = c + 3 + 8 * (j - 1);
                const bool a3 = (j == 2 || j == 5);
                const float s = fmaf(q[0], x, fmaf(q[1], y, fmaf(q[2], z, q[3])));
                const float A = ((q[7] + fmaf(q[6], z, a3 ? t3z : t1z)) + fmaf(q[5], y, a3 ? t3y : t1y)) +
                                fmaf(q[4], x, a3 ? t3x : t1x);
                hex_frac(s, A, es, ea, N, D, first, zero);
            }
        }
        const float v = first ? FLT_MAX : __fdividef(N, D);
        float m = v;
        if (P == 32) m = redux_min(v);
        else for (int o = P >> 1; o; o >>= 1) m = fminf(m, __shfl_xor_sync(FULL, m, o));
        const unsigned zeros = __ballot_sync(FULL, zero);
        const unsigned near = __ballot_sync(FULL, !first && (!(v > m + fabsf(m) * 0x1p-19f) || !(D < 1e36f)));
        const int base = lane & ~(P - 1);
        const unsigned group = P == 32 ? FULL : ((1u << P) - 1u) << base;
        const int owner = __ffs((int)(near & group)) - 1;
        const float on = __shfl_sync(FULL, N, owner & 31), od = __shfl_sync(FULL, D, owner & 31);
        if (zeros & group) return 0.f;
        if (__popc(near & group) == 1) return on / od;
        return hex_key1(co, k, x, y, z, es, ea);
    }
    // smallest over the touching sub-tets of an upper bound of their key on the level's box
    __device__ __forceinline__ float upper(const QuadLevel& lv, int lane) const {
        const float dd = fmaf(lv.dx, lv.dx, fmaf(lv.dy, lv.dy, lv.dz * lv.dz));
        float best = FLT_MAX;
        for (int i = lane; i < 6 * k; i += 32) {
            if (constant(i)) continue;
            float4 A, B;
            float alpha;
            load(i, A, B, alpha);
            const float det = fmaf(A.z, lv.dz, fmaf(A.y, lv.dy, fmaf(A.x, lv.dx, A.w)));
            const float L = fmaf(alpha, dd, fmaf(B.z, lv.dz, fmaf(B.y, lv.dy, fmaf(B.x, lv.dx, B.w))));
            const float dD = fmaf(fabsf(A.x), lv.Sx, fmaf(fabsf(A.y), lv.Sy, fabsf(A.z) * lv.Sz));
            const float dL = fmaf(fabsf(fmaf(2.f * alpha, lv.dx, B.x)), lv.Sx,
                                  fmaf(fabsf(fmaf(2.f * alpha, lv.dy, B.y)), lv.Sy, fabsf(fmaf(2.f * alpha, lv.dz, B.z)) * lv.Sz));
            // with the roundings of det and L, both far below 2^-18 of the magnitudes that enter them
            const float Xm = fabsf(lv.dx) + lv.Sx, Ym = fabsf(lv.dy) + lv.Sy, Zm = fabsf(lv.dz) + lv.Sz;
            const float eD = 0x1p-18f * fmaf(fabsf(A.x), Xm, fmaf(fabsf(A.y), Ym, fmaf(fabsf(A.z), Zm, fabsf(A.w))));
            const float eL = 0x1p-18f * fmaf(fabsf(B.x), Xm, fmaf(fabsf(B.y), Ym, fmaf(fabsf(B.z), Zm, fabsf(B.w) + alpha * dd)));
            const float hi = (det + dD) + eD, lo = (L - dL) - eL;
            float u = FLT_MAX;
            if (lo > 0.f) u = hi > 0.f ? __fdividef(hi * hi, (lo * lo) * lo) * (1.f + 0x1p-13f) : 0.f;
            if (u >= 0.f) best = fminf(best, u);
        }
        return redux_min(best);
    }
};

// Keys are a minimum over the items, in whatever order they are folded, only while every A is positive and the
// products of the fold are normal numbers. The thresholds es and ea see to that where the ring's extent is
// about 1, but they shrink with a growing extent, and NaN positions make the fold depend on the order. Whether
// a halfhex (coefficients c, box half-extents X, Y, Z) has such an item: a constant part with a small A, or a
// sub-tet whose A is bounded above 2^-12 neither where its gradient vanishes nor by its tangent at the origin.
static __device__ __forceinline__ bool hex_odd(const float* __restrict__ c, float X, float Y, float Z) {
    bool odd = !(c[1] > 0x1p-36f) || c[0] != c[0];
#pragma unroll 1
    for (int j = 0; j < 5; ++j) {
        const float* q = c + 3 + 8 * j;
        const float least = fmaf((j == 1 || j == 4) ? -1.f / 12.f : -0.25f, fmaf(q[4], q[4], fmaf(q[5], q[5], q[6] * q[6])), q[7]);
        const float tangent = q[7] - fmaf(fabsf(q[4]), X, fmaf(fabsf(q[5]), Y, fabsf(q[6]) * Z));
        if (!(fmaxf(least, tangent) > 0x1p-12f) || q[3] != q[3]) odd = true;
    }
    return odd;
}

// All candidates of a level by hex_key1, eight (four) along x at a time: they share the loads and what depends on y and
// z, and their folds are independent chains. By one warp, or by warp w of a team of four, a quarter each: the
// largest key and, on ties, the lowest linear index, on every lane of the warp; NaN keys never win.
template <int W>
static __device__ __noinline__ float2 hex_level(const float* __restrict__ co, int k, float es, float ea, QuadLevel lv, int w) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NX = W == 1 ? 8 : 4;
    const int lane = threadIdx.x & 31, x0 = W == 1 ? 0 : 4 * (w & 1);
    float bk = -FLT_MAX;
    int bi = 1 << 30;
    const float y = fmaf(grid_offset(lane & 7), lv.Sy, lv.dy), t1y = y * y, t3y = (3.f * y) * y;
    float x[NX], t1x[NX], t3x[NX];
#pragma unroll
    for (int i = 0; i < NX; ++i) {
        x[i] = fmaf(grid_offset(x0 + i), lv.Sx, lv.dx);
        t1x[i] = x[i] * x[i];
        t3x[i] = (3.f * x[i]) * x[i];
    }
#pragma unroll 1
    for (int part = W == 1 ? 0 : w >> 1; part < (W == 1 ? 2 : (w >> 1) + 1); ++part) {
        const int zi = (lane >> 3) + 4 * part;
        const float z = fmaf(grid_offset(zi), lv.Sz, lv.dz), t1z = z * z, t3z = (3.f * z) * z;
        float N[NX], D[NX];
        unsigned zero = 0;
#pragma unroll
        for (int i = 0; i < NX; ++i) { N[i] = co[0]; D[i] = co[1]; }
#pragma unroll 1
        for (int h = 0; h < k; ++h) {
            const float* c = co + HEX_CO * h;
            const float cn = c[0], cd = c[1];
            if (c[2] != 0.f) zero = 0xffu;
#pragma unroll
            for (int i = 0; i < NX; ++i) {
                const bool less = h > 0 && cn * D[i] < N[i] * cd;
                N[i] = less ? cn : N[i];
                D[i] = less ? cd : D[i];
            }
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                const float* q = c + 3 + 8 * j;
                const bool a3 = (j == 1 || j == 4);
                const float sY = fmaf(q[1], y, fmaf(q[2], z, q[3]));
                const float aY = (q[7] + fmaf(q[6], z, a3 ? t3z : t1z)) + fmaf(q[5], y, a3 ? t3y : t1y);
#pragma unroll
                for (int i = 0; i < NX; ++i) {
                    const float s = fmaf(q[0], x[i], sY);
                    const float A = aY + fmaf(q[4], x[i], a3 ? t3x[i] : t1x[i]);
                    const bool null = s < es || A < ea;   // the key is zero, whatever the fold holds
                    const float num = s * s, den = (A * A) * A;
                    const bool less = num * D[i] < N[i] * den;
                    zero |= null ? 1u << i : 0u;
                    N[i] = less ? num : N[i];
                    D[i] = less ? den : D[i];
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NX; ++i) {
            const float key = (zero >> i) & 1u ? 0.f : N[i] / D[i];
            const int idx = x0 + i + 8 * (lane & 7) + 64 * zi;
            if (key > bk || (key == bk && idx < bi)) { bk = key; bi = idx; }
        }
    }
    const float best = redux_max(bk);
    bi = (int)__reduce_min_sync(FULL, bk == best ? (unsigned)bi : 1u << 30);
    return make_float2(best, __int_as_float(bi));
}

// What a team of four warps per vertex shares: the first one searches, the others wait for levels to be evaluated in full
struct HexTeam {
    QuadLevel lv;
    float es, ea;
    int k, go;
    float2 best[4];
};

// the other warps' loop; every barrier pairs with one of hex_team_level or, with go = 0, of the end
static __device__ __forceinline__ void hex_team_help(HexTeam* team, const float* __restrict__ co, int w) {
    while (true) {
        __syncthreads();
        if (!team->go) return;
        const float2 r = hex_level<4>(co, team->k, team->es, team->ea, team->lv, w);
        if ((threadIdx.x & 31) == 0) team->best[w] = r;
        __syncthreads();
    }
}

static __device__ __forceinline__ float2 hex_team_level(HexTeam* team, const float* __restrict__ co, int k, float es, float ea, const QuadLevel& lv) {
    if ((threadIdx.x & 31) == 0) {
        team->lv = lv;
        team->es = es; team->ea = ea; team->k = k; team->go = 1;
    }
    __syncthreads();
    float2 best = hex_level<4>(co, k, es, ea, lv, 0);
    __syncthreads();
#pragma unroll
    for (int w = 1; w < 4; ++w) {
        const float2 r = team->best[w];
        if (r.x > best.x || (r.x == best.x && __float_as_int(r.y) < __float_as_int(best.y))) best = r;
    }
    __syncwarp();
    return best;
}

// Search from the local origin; returns whether the vertex moved. scratch: TS_WARP_BYTES of the warp,
// subset: 6 k places.
// odd: every level in full (hex_odd). W: warps of the team (1: no team).
template <int W>
static __device__ __forceinline__ bool hex_plain_search(HexItems ring, bool odd, HexTeam* team, float* __restrict__ scratch,
                                                        unsigned short* __restrict__ subset, float sx, float sy, float sz,
                                                        float grid_scale, int depth, int lane, float& dx, float& dy,
                                                        float& dz) {
    constexpr unsigned FULL = 0xffffffffu;
    unsigned short* list = reinterpret_cast<unsigned short*>(scratch + TS_TABLE);
    const float off = grid_offset(lane & 7);
    dx = 0.f; dy = 0.f; dz = 0.f;
    // the constant key Q, folded in ring order
    float N = 0.f, D = 1.f;
    for (int h = 0; h < ring.k; ++h) {
        const float* c = ring.co + HEX_CO * h;
        if (c[2] != 0.f) return false;   // every key is zero
        if (h == 0 || c[0] * D < N * c[1]) { N = c[0]; D = c[1]; }
    }
    const float Q = N / D;
    float qLast = odd ? hex_key1(ring.co, ring.k, 0.f, 0.f, 0.f, ring.es, ring.ea) : ring.group_key(0.f, 0.f, 0.f, 32, lane);
    bool moved = false, full = odd;   // once a level is evaluated in full, so are the smaller ones
    float ds = grid_scale;
    for (int level = 0; level < depth; ++level) {
        QuadLevel lv{dx, dy, dz, ds * sx, ds * sy, ds * sz, 0.f, 0.f, 0.f, false};
        ds = ds * (2.0f / 7.0f);
        if (lv.Sx == 0.f && lv.Sy == 0.f && lv.Sz == 0.f) continue;   // a lattice: every candidate is the centre
        float bk = -FLT_MAX;
        int bi = 1 << 30;
        if (!full) {
            const float U = fminf(ring.upper(lv, lane), Q);
            const float clear_of_U = U + (U * 0x1p-13f + 1e-37f);
            if (clear_of_U < qLast) continue;   // nothing on the box can beat the current key
            lv.sq2 = sqrt_approx(clear_of_U) * (1.f + 0x1p-20f);
            lv.ties = U == Q;
            const float thr = key_below(fminf(qLast, U));
            if (thr > 0.f) lv.sq = sqrt_approx(thr) * (1.f - 0x1p-20f);
            else lv.low = ring.es * 0.999f;   // a key above zero needs det >= es
            float s[16], rho, above;
            quad_filter<HexItems, true, false>(ring, lv, scratch, lane, s, rho, above, subset, ring.m);
            ring.subset = subset;
            const bool ties = lv.ties && above < FLT_MAX;   // candidates clearly above have the key Q
            float cut = 0.f;
            unsigned clear = ties ? at_least(s, above) : 0u;
            if (qLast < Q) {
                int place;
                const float top = top_candidate(s, bi, place);
                if (top < 0.f) continue;   // every candidate is dropped
                if (top >= 0.f) {
                    const float3 c = grid_candidate(bi, off, lv);
                    bk = ring.m > 8 ? ring.group_key(c.x, c.y, c.z, 32, lane) : ring.key(c.x, c.y, c.z);
                    if (thr > 0.f && bk > qLast) cut = (sqrt_approx(key_below(bk)) * (1.f - 0x1p-20f) - lv.sq) * (rho * 0.999f);
                    if (!(cut > 0.f)) cut = 0.f;
                } else {
                    bi = 1 << 30;
                }
                if (ties) {
                    int low = 1 << 30;
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (clear & (0x8000u >> i)) low = min(low, grid_index(lane, i));
                    low = (int)__reduce_min_sync(FULL, (unsigned)low);
                    if (low < 512 && (Q > bk || (Q == bk && low < bi))) { bk = Q; bi = low; }
                }
            }
            const unsigned alive = at_least(s, cut) & ~clear;
            // Boxes that shrink with the smallest ring distance can leave every candidate within the margins: judged one per
            // lane, a round of 32 candidates over the whole ring takes about half as long as all of them in full, and longer
            // than a team of four takes for that (lattice with 1 % of jitter, 12^3 cells, us per iteration with the
            // factor 2 / 4 / 7: 381 / 494 / 568; jittered 16^3 396 / 464 / 467).
            full = ((__reduce_add_sync(FULL, __popc(alive)) + 31) >> 5) * ring.m > (W == 1 ? 14 : 2) * ring.k;
            if (!full) judge(ring, lv, alive, off, list, lane, bk, bi);
        }
        if (full) {
            const float2 best = W == 1 ? hex_level<1>(ring.co, ring.k, ring.es, ring.ea, lv, 0) : hex_team_level(team, ring.co, ring.k, ring.es, ring.ea, lv);
            bk = best.x;
            bi = __float_as_int(best.y);
        }
        if (bi < 512 && qLast < bk) {
            const float3 c = grid_candidate(bi, off, lv);
            dx = c.x; dy = c.y; dz = c.z;
            qLast = bk;
            moved = true;
        }
    }
    return moved;
}

}  // namespace vsdmo
