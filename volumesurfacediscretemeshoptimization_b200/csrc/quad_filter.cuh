// quad_filter.cuh -- exact candidate filter of the volume searches: lower bounds on how far each of
// the 8 x 8 x 8 candidates of a level lies above a ring key, one warp per vertex.
//
// A ring is a set of items (the tets of a vertex, or the sub-tets of its hexahedra that touch it)
// with a determinant det(p) affine in the candidate p and a sum of squared edges L(p) = .. + alpha
// |p|^2, and the item's key is det^2 / L^3. A level can only move the vertex to a candidate whose
// ring key (the smallest item key) beats the current key q, so a candidate for which any item's key
// lies below q can be dropped. For q > 0 the condition det^2 / L^3 >= thr (thr just below q) is
// det >= sqrt(thr) L^(3/2), and L^(3/2) is convex in L: its tangent T(L) = 1.5 r L - 0.5 r^3 at r^2
// lies below it for every r, so
//     g(p) = w (det(p) - sqrt(thr) T(L(p))) >= 0
// holds for every candidate that can beat q (w > 0 scales the item, about 1 / r^3). det is affine
// and L an isotropic quadratic in p, so g splits into a sum of one function per axis: on the
// separable grid it is a table look-up and two additions per (candidate, item), and the z additions
// run two at a time (f32x2) with one three-operand minimum per two items. For thr <= 0 the condition
// is det(p) >= low and the same form holds without the quadratic part.
//
// Pruning by one exact key. The smallest g of a candidate estimates how far its ring key's root
// exceeds sqrt(thr), so the candidate of the largest is judged first. When its key K1 beats q, a
// candidate that beats K1 needs det >= sqrt(thr1) T(L) with thr1 just below K1, hence
//     g(p) >= (sqrt(thr1) - sqrt(thr)) w T(L(p)) >= (sqrt(thr1) - sqrt(thr)) rho,
// rho the smallest w T over the box and the items.
//
// The filter is exact: g is evaluated with its own roundings, so every item's constant is raised by
// 2^-18 of the sum of the magnitudes that enter it, far above the few 2^-24 that det, L and g can be
// off by; an overflow makes that term infinite or NaN, and a candidate is only dropped for a sum
// that compares below the limit.
#pragma once
#include "f32x2.cuh"
#include <cfloat>

namespace vsdmo {

// floats per item: (x_i, x_i) for i = 0..7, (y_j, y_j, y_7-j, y_7-j) for j = 0..3, z at places 0 1 2 3
// 7 6 5 4; 44: no bank conflicts
constexpr int TS_SLOT = 44;
constexpr int TS_TABLE = 32 * TS_SLOT;      // up to 32 items between two looks at the candidates
// Items looked at first (rings of up to 32 items) and the pruning bound below which the others follow, when
// anything survives: 6 / 8 / 10 / 12 / all tets first took 0.479 / 0.418 / 0.404 / 0.409 / 0.439 ms
// per iteration of the 48^3 cube (20 iterations), never looking at the others 0.418 (10 tets).
constexpr int TS_CRIT = 10;
constexpr float TS_RHO = 0.3f;
constexpr int TS_LIST = 512;                // survivors (16-bit candidate indices): every candidate fits
// shared memory of one warp's search besides the ring's coefficients, in bytes (a multiple of 16)
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
static __device__ __forceinline__ int grid_index(int lane, int i) {
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

// value just below the key q: what a candidate that beats q cannot fall under on any item (the
// margin covers the rounding of the fraction comparisons along a ring)
static __device__ __forceinline__ float key_below(float q) { return q - (fabsf(q) * 0x1p-14f + 1e-37f); }

// the level a filter looks at: centre, half-extents and the condition's sqrt(thr) and low (one of
// them 0); sq2: WINDOW filters
struct QuadLevel {
    float dx, dy, dz, Sx, Sy, Sz, sq, low, sq2;
    bool ties;
};

// Lower bounds of the 512 candidates centre + offset * S: s[2 q + jj] of a lane is the smallest g of
// candidate grid_index(lane, 2 q + jj) over the items looked at. rho: the smallest w T over the box
// and those items (0 where there is no bound). tab: the warp's TS_TABLE floats. Returns false when
// the items looked at first already drop every candidate (most searches of a nearly converged mesh).
//
// WINDOW (upper: a key that no candidate's ring key exceeds, sq2 the root of a key clearly above it):
//   * above (with lv.ties, which takes every item of the subset into the table): a candidate with
//     s > above has every item's key clearly above upper;
//   * subset, m: the items, in ring order, that are not clearly above upper on the whole box. The
//     others cannot touch any candidate's ring key (the serial fold of fractions ends on the items
//     within rounding of the smallest, whatever the others are), so keys are folded over the subset.
// On the box L^(3/2) <= T(L) + 3/8 dL^2 / sqrt(Lmin), so g exceeds w (det - sq2 L^(3/2)) by at most
// over = (sq2 - sq) w Tmax + sq2 w 3/8 dL^2 / sqrt(Lmin) + twice the allowance. An item that may fall
// under the ring's lower limits of det or L on the box is never clearly above.
//
// ONE: the ring has at most 32 items. Bound: issue; 21 slots per item and 16 candidates. Items whose g
// is positive on the whole box are left out before the loop.
template <class Ring, bool WINDOW, bool ONE>
static __device__ __forceinline__ bool quad_filter(const Ring& ring, const QuadLevel& lv, float* __restrict__ tab, int lane,
                                                   float (&s)[16], float& rho, float& above,
                                                   unsigned short* __restrict__ subset, int& m) {
    constexpr unsigned FULL = 0xffffffffu;
    const float Xm = fabsf(lv.dx) + lv.Sx, Ym = fabsf(lv.dy) + lv.Sy, Zm = fabsf(lv.dz) + lv.Sz;
    const float R2 = fmaf(Xm, Xm, fmaf(Ym, Ym, Zm * Zm));
    const float dd = fmaf(lv.dx, lv.dx, fmaf(lv.dy, lv.dy, lv.dz * lv.dz));
#pragma unroll
    for (int i = 0; i < 16; ++i) s[i] = FLT_MAX;
    rho = FLT_MAX;
    above = 0.f;
    m = 0;
    const int n = ring.items();
    const unsigned lower = (1u << lane) - 1u;
    int t0 = 0;
    do {
        // the table takes the items of up to 32 lanes that drop a candidate
        int base = 0, first = 0;
        do {
            float4 A, B;
            float alpha;
            ring.load(min(t0 + lane, n - 1), A, B, alpha);
            // the tangent's point r^2 = L and its slope b = 1.5 sqrt(thr) r, all scaled by w
            const float det = fmaf(A.z, lv.dz, fmaf(A.y, lv.dy, fmaf(A.x, lv.dx, A.w)));
            const float L = fmaf(alpha, dd, fmaf(B.z, lv.dz, fmaf(B.y, lv.dy, fmaf(B.x, lv.dx, B.w))));
            const float r = sqrt_approx(fmaxf(L, 0.f));
            const float r3 = (r * r) * r;
            const float w = __fdividef(1.f, r3);
            const float b = 1.5f * (lv.sq * r), a = 0.5f * (lv.sq * r3);
            // magnitudes of all that enters g, for the rounding allowance
            const float magL = fmaf(fabsf(B.x), Xm, fmaf(fabsf(B.y), Ym, fmaf(fabsf(B.z), Zm, fmaf(alpha, R2, fabsf(B.w)))));
            const float mag = fmaf(fabsf(A.x), Xm, fmaf(fabsf(A.y), Ym, fmaf(fabsf(A.z), Zm, fabsf(A.w)))) +
                              fmaf(b, magL, a + fabsf(lv.low));
            const float slack = 0x1p-18f * mag;
            const float g = w * (((det - lv.low) + fmaf(-b, L, a)) + slack);
            const float a2 = 2.f * alpha;   // gradient of L
            const float Lx = fmaf(a2, lv.dx, B.x), Ly = fmaf(a2, lv.dy, B.y), Lz = fmaf(a2, lv.dz, B.z);
            const float wx = w * lv.Sx, wy = w * lv.Sy, wz = w * lv.Sz, ab = alpha * b;
            const float Px = wx * fmaf(-b, Lx, A.x), Qx = ab * (lv.Sx * wx);
            const float Py = wy * fmaf(-b, Ly, A.y), Qy = ab * (lv.Sy * wy);
            const float Pz = wz * fmaf(-b, Lz, A.z), Qz = ab * (lv.Sz * wz);
            // L >= L(centre) - sum |grad L| S on the box
            const float dL = fmaf(fabsf(Lx), lv.Sx, fmaf(fabsf(Ly), lv.Sy, fabsf(Lz) * lv.Sz));
            const float Lmin = L - dL;
            // an item whose g is positive on the whole box (concave per axis: smallest at an end) drops nothing
            const float gmin = g - (((fabsf(Px) + Qx) + (fabsf(Py) + Qy)) + (fabsf(Pz) + Qz));
            const bool in = t0 + lane < n;
            float over = 0.f;
            if constexpr (WINDOW) {
                const float dm = fmaf(alpha, fmaf(lv.Sx, lv.Sx, fmaf(lv.Sy, lv.Sy, lv.Sz * lv.Sz)), dL);
                const float hi = fmaf(1.5f * r, L + dm, -0.5f * r3);
                over = w * fmaf(lv.sq2 - lv.sq, hi, fmaf(lv.sq2, __fdividef(0.375f * (dm * dm), sqrt_approx(Lmin)), 2.f * slack));
                const float dmin = det - fmaf(fabsf(A.x), lv.Sx, fmaf(fabsf(A.y), lv.Sy, fabsf(A.z) * lv.Sz)) - slack;
                const bool valid = Lmin > 0.f && dmin > ring.min_det() && Lmin > ring.min_len() * 1.001f;
                over = valid && over >= 0.f ? fmaf(over, 0x1p-10f, over) : FLT_MAX;
            }
            const unsigned use = __ballot_sync(FULL, in && !(gmin > (lv.ties ? over : 0.f)));
            const int cnt = __popc(use);
            if (!ONE && base + cnt > 32) break;   // these items go into the next table
            if constexpr (WINDOW) {
                const bool near = in && !(gmin > over);
                if (near && !ring.constant(t0 + lane)) above = fmaxf(above, over);
                const unsigned sub = __ballot_sync(FULL, ring.constant(t0 + lane) ? in && ring.keep(t0 + lane, lv.sq2) : near);
                if ((sub >> lane) & 1u) subset[m + __popc(sub & lower)] = (unsigned short)(t0 + lane);
                m += __popc(sub);
            }
            // the items looked at first: the TS_CRIT of smallest det / r^3 (any choice is exact)
            unsigned crit = use;
            if (ONE && cnt > TS_CRIT + 2) {
                const float v = (use >> lane) & 1u ? det * w : FLT_MAX;
                float left = v, top = 0.f;
#pragma unroll
                for (int i = 0; i < TS_CRIT; ++i) {
                    top = redux_min(left);
                    left = left > top ? left : FLT_MAX;
                }
                crit &= __ballot_sync(FULL, !(v > top));
            }
            const int m1 = __popc(crit);
            if ((use >> lane) & 1u) {
                float* u = tab + (base + ((crit >> lane) & 1u ? __popc(crit & lower) : m1 + __popc(use & ~crit & lower))) * TS_SLOT;
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
                const float T = w * fmaf(1.5f * r, fmaf(-0x1p-20f, magL, Lmin), -0.5f * r3);   // less the rounding of Lmin
                rho = fminf(rho, T > 0.f ? T : 0.f);
            }
            first = base + m1;
            base += cnt;
            t0 += 32;
        } while (!ONE && t0 < n);
        // an odd count is padded with an item that drops nothing
        if (base & 1)
            for (int i = lane; i < 40; i += 32) tab[base * TS_SLOT + i] = i < 16 ? FLT_MAX : 0.f;
        if (ONE) rho = redux_min(rho);
        __syncwarp();
        const float* u = tab;
        int j = 0, end = ONE ? first : base;
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
            if (!ONE || j >= base) break;
            if (top_bound(s) < 0.f) return false;
            if (rho >= TS_RHO) break;
            end = base;
        }
        if (!ONE) __syncwarp();   // the table may be rewritten
    } while (!ONE && t0 < n);
    if (!ONE) rho = redux_min(rho);
    if (!(rho < FLT_MAX)) rho = 0.f;   // no item looked at
    if (WINDOW) above = redux_max(above);
    return true;
}

// largest bound of the warp and, when it is not NaN, its candidate (linear index bi; place: lane * 16 +
// bound). The index replaces the low four bits of the bound: an estimate either way.
static __device__ __forceinline__ float top_candidate(const float (&s)[16], int& bi, int& place) {
    constexpr unsigned FULL = 0xffffffffu;
    float e[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) e[i] = __uint_as_float((__float_as_uint(s[i]) & ~15u) | i);
    float top = fmaxf(e[0], e[1]);
#pragma unroll
    for (int i = 2; i < 16; i += 2) top = max3(top, e[i], e[i + 1]);
    const float all = redux_max(top);
    const int owner = __ffs((int)__ballot_sync(FULL, top == all)) - 1;
    const int i = (int)(__float_as_uint(all) & 15u);
    place = owner * 16 + i;
    bi = grid_index(owner, i);
    return all;
}

// bit 15 - i set when bound i is not below the limit
static __device__ __forceinline__ unsigned at_least(const float (&s)[16], float limit) {
    unsigned dead = 0;
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        float u, v;
        upk2(add2(pk2(s[i], s[i + 1]), pk2(-limit, -limit)), u, v);
        dead = __funnelshift_l(__float_as_uint(u), dead, 1);
        dead = __funnelshift_l(__float_as_uint(v), dead, 1);
    }
    return ~dead & 0xffffu;
}

// position of candidate idx; off: grid_offset(lane & 7) of every lane
static __device__ __forceinline__ float3 grid_candidate(int idx, float off, const QuadLevel& lv) {
    constexpr unsigned FULL = 0xffffffffu;
    const float ox = __shfl_sync(FULL, off, idx & 7), oy = __shfl_sync(FULL, off, (idx >> 3) & 7);
    const float oz = __shfl_sync(FULL, off, (idx >> 6) & 7);
    return make_float3(fmaf(ox, lv.Sx, lv.dx), fmaf(oy, lv.Sy, lv.dy), fmaf(oz, lv.Sz, lv.dz));
}

// The candidates set in alive (at_least's bits) judged by their ring key: bk, bi (the same on all
// lanes) become the largest key so far and its candidate, the lowest linear index on ties. Up to 16
// candidates are judged together by 32 / (their number, rounded up to a power of two) lanes each where
// the ring asks for it (a key costs more than splitting it); more go one per lane, 32 at a time. list: TS_LIST places of shared memory.
template <class Ring>
static __device__ __forceinline__ void judge(const Ring& ring, const QuadLevel& lv, unsigned alive, float off,
                                             unsigned short* __restrict__ list, int lane, float& bk, int& bi) {
    constexpr unsigned FULL = 0xffffffffu;
    const int cnt = __popc(alive);
    if (!__any_sync(FULL, cnt)) return;
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
        list[at++] = (unsigned short)grid_index(lane, 15 - bit);
    }
    __syncwarp();
    if (total <= 16 && ring.groups()) {
        const int P = total <= 1 ? 32 : total <= 2 ? 16 : total <= 4 ? 8 : total <= 8 ? 4 : 2;
        const int idx = list[min(lane / P, total - 1)];
        const float3 c = grid_candidate(idx, off, lv);
        const float key = ring.group_key(c.x, c.y, c.z, P, lane);
        if (key > bk || (key == bk && idx < bi)) { bk = key; bi = idx; }
    } else {
        for (int j = lane; j - lane < total; j += 32) {
            const int idx = list[min(j, total - 1)];
            const float3 c = grid_candidate(idx, off, lv);
            const float key = ring.key(c.x, c.y, c.z);
            if (key > bk || (key == bk && idx < bi)) { bk = key; bi = idx; }
        }
    }
    const float best = redux_max(bk);
    bi = (int)__reduce_min_sync(FULL, bk == best ? (unsigned)bi : 1u << 30);
    bk = best;
    __syncwarp();   // the list may be rewritten
}

}  // namespace vsdmo
