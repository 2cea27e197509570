// flat_search.cuh -- the 8 x 8 hierarchical 2D search of four vertices per warp, eight lanes each.
//
// Same result as the 32-thread search of k_optimizeHierarchical2DFlat
// (dmo/DMOTriFlatImplCub.h:24-152): virtual thread t = 8 (i & 3) + j owns candidates (i, j) and
// (i + 4, j) of the level, keeps the second on a tie, the first thread of the largest key wins, the
// vertex moves to it when it beats the current key, and it is written when the last level's largest
// key beats the start's. Keys are the exact operations of the ring fold: the fraction A / L of every
// ring element with A affine and L quadratic in the candidate; negative areas and corners as in bkey.
//
// Exact candidate filter, as in quad_filter.cuh: a candidate that beats the key q has A - q L >= 0 on
// every element, and that is already a sum of one function per axis. Lane j of a group tabulates the
// x parts of every element at x_j, then adds its y part to all eight: one packed addition and one
// three-operand minimum per two candidates and two elements. Each element's constant is raised by
// 2^-18 of the magnitudes that enter it. The candidate of the largest bound is judged first (its ring
// elements spread over the group's lanes); a candidate that beats its key K1 needs
// w (A - q L) >= (K1 - q) rho, rho the smallest w L on the box (w = 1 / L at the vertex), which leaves
// a candidate or two for the full key.
//
// Bound: issue (66 % of the slots on 256 mixed meshes). The search with a warp per vertex spends most of
// its slots on the idle lanes of a six-element ring and on reductions per vertex: 8.35 ms per
// iteration of 256 meshes (3.2 M vertices), this one 2.28 ms, and 2.35 ms with the rings searched apart
// (their code costs the kernel registers). Loops over the ring are not unrolled: unrolled by four they
// overflowed the instruction cache (3.46 ms, half the stalls instruction fetches).
#pragma once
#include "f32x2.cuh"
#include "flat_key.cuh"
#include <cfloat>

namespace vsdmo {

constexpr int F8_MAX_RING = 16;   // larger rings take the general search
// floats of shared memory per group: 12 per element exact coefficients, 8 filter coefficients, 16 of ring
// positions and tables; the remainder keeps the four groups of a warp in different banks
__host__ __device__ constexpr int f8_group_floats(int maxk) { return 36 * maxk + ((8 - 36 * maxk) & 31); }

template <int FK>
struct F8 {
    static constexpr int CS = FK == 3 ? 8 : 12;   // floats per element
    // exact coefficients of ring element t at c
    static __device__ __forceinline__ void coeffs(float ax, float ay, float bx, float by, float cx, float cy, float* c) {
        if (FK == 3) btri_co(ax, ay, cx, cy, c);
        else bquad_co(ax, ay, bx, by, cx, cy, c);
    }
    // value and edge sum of element t; neg: a quad corner turns clockwise
    static __device__ __forceinline__ void eval(const float* c, float x, float y, float tx, float ty, float& A, float& L, bool& neg) {
        const float4 u = *reinterpret_cast<const float4*>(c), v = *reinterpret_cast<const float4*>(c + 4);
        if (FK == 3) {
            A = fmaf(u.y, y, fmaf(u.x, x, u.z));
            L = (v.y + fmaf(u.w, x, tx)) + fmaf(v.x, y, ty);
        } else {
            const float c8 = c[8];
            const float c1 = fmaf(u.y, y, fmaf(u.x, x, u.z));
            const float c2 = fmaf(v.x, y, fmaf(u.w, x, v.y));
            neg |= c1 < 0.f || c2 < 0.f;
            A = c1 + c2;
            L = (c8 + fmaf(v.z, x, tx)) + fmaf(v.w, y, ty);
        }
    }
    // ring key of (x, y), serial
    static __device__ __forceinline__ float key(const float* co, int k, float x, float y) {
        const float tx = (2.0f * x) * x, ty = (2.0f * y) * y;
        float N = 0.f, D = 1.f, amin = 0.f;
        bool neg = false;
#pragma unroll 1
        for (int t = 0; t < k; ++t) {
            float A, L;
            eval(co + CS * t, x, y, tx, ty, A, L, neg);
            if (t == 0) { N = A; D = L; amin = A; continue; }
            if (A * D < N * L) { N = A; D = L; }
            if (FK == 3) amin = fminf(amin, A);
        }
        if (FK == 3) return amin < 0.f ? amin : N / D;
        return neg ? -1.f : N / D;
    }
    // the same key by the group's lanes: every lane folds every eighth element; lanes within 2^-19 of the
    // smallest fold repeat the serial one
    static __device__ __forceinline__ float group_key(const float* co, int k, float x, float y, int lane) {
        constexpr unsigned FULL = 0xffffffffu;
        const int gl = lane & 7, g0 = lane & 24;
        const float tx = (2.0f * x) * x, ty = (2.0f * y) * y;
        float N = 0.f, D = 1.f, amin = 0.f;
        bool neg = false;
#pragma unroll 1
        for (int t = gl; t < k; t += 8) {
            float A, L;
            eval(co + CS * t, x, y, tx, ty, A, L, neg);
            if (t == gl) { N = A; D = L; amin = A; continue; }
            if (A * D < N * L) { N = A; D = L; }
            amin = fminf(amin, A);
        }
        const float v = gl >= k ? FLT_MAX : FK == 3 && amin < 0.f ? amin : __fdividef(N, D);
        float m = v;
#pragma unroll
        for (int o = 4; o; o >>= 1) m = fminf(m, __shfl_xor_sync(FULL, m, o));
        const unsigned near = __ballot_sync(FULL, gl < k && (!(v > m + fabsf(m) * 0x1p-19f) || !(D < 1e36f)));
        const unsigned negs = __ballot_sync(FULL, neg);
        const unsigned group = 0xffu << g0;
        const int owner = __ffs((int)(near & group)) - 1;
        const float on = __shfl_sync(FULL, N, owner & 31), od = __shfl_sync(FULL, D, owner & 31);
        if (FK == 3 && m < 0.f) return m;
        if (FK == 4 && (negs & group)) return -1.f;
        if (__popc(near & group) == 1) return on / od;
        return key_again(co, k, x, y);
    }
    static __device__ __noinline__ float key_again(const float* co, int k, float x, float y) { return key(co, k, x, y); }
};

// One vertex per group of eight lanes (on: the group has one). sm: the group's f8_group_floats(maxk).
// All lanes of the warp call this together.
//
// Keys are a minimum only while every edge sum L is positive: at a candidate on (or, with the rounding of
// L, beside) two coincident ring points the fold meets 0 / 0 or a negative L and its result depends on
// the order of the elements, and so it does with NaN positions. Rings in which L is not bounded well
// above its rounding (2^-15 of the magnitudes that enter it, on the whole search box) are searched apart, by
// the steps of the general search of L lanes on the coefficients at hand.
template <int FK, bool COHERENT>
__device__ void flat_search8(float4* __restrict__ pos, const int* __restrict__ rowptr, const int4* __restrict__ he, int v,
                             bool on, float gs, int depth, float* __restrict__ sm, int maxk, int lane, int L) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int CS = F8<FK>::CS;
    const int gl = lane & 7, g0 = lane & 24;
    const unsigned group = 0xffu << g0;
    float* co = sm;                                        // exact coefficients
    float4* fc = reinterpret_cast<float4*>(sm + 12 * maxk);   // filter coefficients, 2 per element
    float* tab = sm + 20 * maxk;
    float2* ring = reinterpret_cast<float2*>(tab);         // setup only
    int b = 0, k = 0;
    float4 c0 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (on) {
        b = rowptr[v];
        k = rowptr[v + 1] - b;
        if (k > maxk) k = 0;
        c0 = ldpos<COHERENT>(pos + v);
    }
    float mdx = 0.f, mdy = 0.f;
#pragma unroll 1
    for (int t = gl; t < k; t += 8) {
        const int4 h = he[b + t];
        const float4 p = ldpos<COHERENT>(pos + h.x);
        const float px = p.x - c0.x, py = p.y - c0.y;
        mdx = fmaxf(mdx, fabsf(px)); mdy = fmaxf(mdy, fabsf(py));
        ring[t] = make_float2(px, py);
        if (FK == 4) {
            const float4 p2 = ldpos<COHERENT>(pos + he[h.w].x);
            const float qx = p2.x - c0.x, qy = p2.y - c0.y;
            mdx = fmaxf(mdx, fabsf(qx)); mdy = fmaxf(mdy, fabsf(qy));
            ring[maxk + t] = make_float2(qx, qy);
        }
    }
    __syncwarp();
#pragma unroll
    for (int o = 4; o; o >>= 1) {
        mdx = fmaxf(mdx, __shfl_xor_sync(FULL, mdx, o));
        mdy = fmaxf(mdy, __shfl_xor_sync(FULL, mdy, o));
    }
    const float mm = fmaxf(mdx, mdy);
    if (!(mm > 0.f) || !(mm < FLT_MAX)) k = 0;
    const int kmax = __reduce_max_sync(FULL, k);
    if (kmax == 0) return;
    int ex;
    (void)frexpf(mm, &ex);
    const float ps = bexp2(-ex);
    const float sx = bscale(mdx, ps, -ex), sy = bscale(mdy, ps, -ex);
    bool odd = false;
    // the levels' half-extents sum to at most 1.4 gs
    const float Xm = (1.5f * gs) * sx, Ym = (1.5f * gs) * sy;
#pragma unroll 1
    for (int t = gl; t < k; t += 8) {
        const float2 a = ring[t], n = ring[t + 1 == k ? 0 : t + 1];
        float2 c = a;
        if (FK == 4) c = ring[maxk + t];
        float K[12];
        F8<FK>::coeffs(bscale(a.x, ps, -ex), bscale(a.y, ps, -ex), bscale(c.x, ps, -ex), bscale(c.y, ps, -ex),
                       bscale(n.x, ps, -ex), bscale(n.y, ps, -ex), K);
#pragma unroll
        for (int i = 0; i < (FK == 3 ? 6 : 9); ++i) co[CS * t + i] = K[i];
        float a0, a1, a2, l0, l1, l2, ma;
        if (FK == 3) {
            a0 = K[0]; a1 = K[1]; a2 = K[2]; l0 = K[3]; l1 = K[4]; l2 = K[5];
            ma = fmaf(fabsf(a0), Xm, fmaf(fabsf(a1), Ym, fabsf(a2)));
        } else {
            a0 = K[0] + K[3]; a1 = K[1] + K[4]; a2 = K[2] + K[5]; l0 = K[6]; l1 = K[7]; l2 = K[8];
            ma = fmaf(fabsf(K[0]) + fabsf(K[3]), Xm, fmaf(fabsf(K[1]) + fabsf(K[4]), Ym, fabsf(K[2]) + fabsf(K[5])));
        }
        const float w = __fdividef(1.f, l2);
        const float ml = fmaf(fabsf(l0), Xm, fmaf(fabsf(l1), Ym, fmaf(2.f * Xm, Xm, fmaf(2.f * Ym, Ym, l2))));
        // L is smallest where its gradient vanishes; where that is too small, on the part of the box nearest to the corners
        const float least = fmaf(-0.125f, fmaf(l0, l0, l1 * l1), l2), limit = 0x1p-15f * fmaxf(ml, 0x1p-10f);
        if (!(least > limit)) {
            const float ax = fmaxf(fabsf(bscale(a.x, ps, -ex)) - Xm, 0.f), ay = fmaxf(fabsf(bscale(a.y, ps, -ex)) - Ym, 0.f);
            const float nx = fmaxf(fabsf(bscale(n.x, ps, -ex)) - Xm, 0.f), ny = fmaxf(fabsf(bscale(n.y, ps, -ex)) - Ym, 0.f);
            if (least != least || !((ax * ax + ay * ay) + (nx * nx + ny * ny) > limit)) odd = true;
        }
        fc[2 * t] = make_float4(w * a0, w * a1, w * a2, w * l0);
        fc[2 * t + 1] = make_float4(w * l1, w, (0x1p-18f * w) * ma, (0x1p-18f * w) * ml);
    }
    __syncwarp();
    for (unsigned apart = __ballot_sync(FULL, odd); apart;) {
        const int first = (__ffs((int)apart) - 1) & 24;
        apart &= ~(0xffu << first);
        const float* c = co + ((first - g0) >> 3) * f8_group_floats(maxk);
        const int n = __shfl_sync(FULL, k, first);
        const float fx = __shfl_sync(FULL, sx, first), fy = __shfl_sync(FULL, sy, first);
        const float q0 = F8<FK>::key_again(c, n, 0.f, 0.f);
        float mx = 0.f, my = 0.f, ql = q0, top = -FLT_MAX, h = gs;
#pragma unroll 1
        for (int level = 0; level < depth; ++level) {
            float bv = -FLT_MAX, bx = 0.f, by = 0.f;
            int bt = 1 << 30;
#pragma unroll 1
            for (int t = lane; t < 32 && lane < L; t += L) {
                const float x1 = fmaf(boffset(t >> 3, 8), h * fx, mx), x2 = fmaf(boffset((t >> 3) + 4, 8), h * fx, mx);
                const float y = fmaf(boffset(t & 7, 8), h * fy, my);
                const float q1 = F8<FK>::key_again(c, n, x1, y), q2 = F8<FK>::key_again(c, n, x2, y);
                const float val = q2 > q1 ? q2 : q1;
                if (bt == (1 << 30) || val > bv) { bv = val; bt = t; bx = q1 > q2 ? x1 : x2; by = y; }
            }
#pragma unroll 1
            for (int o = L >> 1; o; o >>= 1) {
                const float ov = __shfl_xor_sync(FULL, bv, o), ox = __shfl_xor_sync(FULL, bx, o), oy = __shfl_xor_sync(FULL, by, o);
                const int ot = __shfl_xor_sync(FULL, bt, o);
                if (ov > bv || (ov == bv && ot < bt)) { bv = ov; bt = ot; bx = ox; by = oy; }
            }
            if (ql < bv) { mx = bx; my = by; ql = bv; }
            top = bv;
            h = h * (2.0f / 7.0f);
        }
        // NaN keys may leave the lanes with different winners: the first one's counts
        mx = __shfl_sync(FULL, mx, 0);
        my = __shfl_sync(FULL, my, 0);
        const int better = __shfl_sync(FULL, q0 < top ? 1 : 0, 0);
        if (lane == first && better) {
            const float pu = bexp2(ex);
            pos[v] = make_float4(c0.x + bscale(mx, pu, ex), c0.y + bscale(my, pu, ex), c0.z, c0.w);
        }
        if (g0 == first) k = -1;
    }
    const float off = boffset(gl, 8);   // offset i of an axis is lane i's of the group
    float dx = 0.f, dy = 0.f, ds = gs;
    float qOld = 0.f, qLast = 0.f;
    bool write = false;
    // level -1 takes the start's key
    for (int level = -1; level < depth; ++level) {
        const float Sx = level < 0 ? 0.f : ds * sx, Sy = level < 0 ? 0.f : ds * sy;
        float s[8], cut = 0.f, all = 0.f, below = 0.f, q = 0.f, rho = FLT_MAX;
        int pi = 0, pj = 0;
        const bool last = level == depth - 1;
        float yg = 0.f;
        if (level >= 0) {
            ds = ds * (2.0f / 7.0f);
            const float base = last ? qOld : qLast;   // the last level decides the write against the start's key
            below = base - (fabsf(base) * 0x1p-14f + 1e-37f);
            q = fmaxf(below, 0.f);
            const float low = FK == 3 ? fminf(below, 0.f) : 0.f;
            const bool corners = FK == 4 && base < 0.f;   // a quad ring with a clockwise corner: no corner may be
            const float xg = fmaf(off, Sx, dx);
            yg = fmaf(off, Sy, dy);
#pragma unroll 1
            for (int t = 0; t < k; ++t) {
                const float4 f = fc[2 * t], e = fc[2 * t + 1];
                if (FK == 4 && corners) {
                    const float* c = co + CS * t;
                    tab[8 * t + gl] = fmaf(e.y * c[0], xg, fmaf(e.y, c[2], e.z));
                    tab[8 * (maxk + t) + gl] = fmaf(e.y * c[3], xg, fmaf(e.y, c[5], e.z));
                } else {
                    const float l = fmaf(f.w, xg, fmaf((2.f * e.y) * xg, xg, 1.f));
                    tab[8 * t + gl] = fmaf(-q, l, fmaf(f.x, xg, f.z)) + fmaf(q, e.w, fmaf(-low, e.y, e.z));
                }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i) s[i] = FLT_MAX;
            if (FK == 4 && corners) {
#pragma unroll 1
                for (int t = 0; t < k; ++t) {
                    const float w = fc[2 * t + 1].y;
                    const float h0 = (w * co[CS * t + 1]) * yg, h1 = (w * co[CS * t + 4]) * yg;
#pragma unroll
                    for (int i = 0; i < 8; ++i) s[i] = min3(s[i], tab[8 * t + i] + h0, tab[8 * (maxk + t) + i] + h1);
                }
            } else {
#pragma unroll 1
                for (int t = 0; t < k; t += 2) {
                    const int u = t + 1 < k ? t + 1 : t;
                    const float4 f0 = fc[2 * t], e0 = fc[2 * t + 1], f1 = fc[2 * u], e1 = fc[2 * u + 1];
                    const float h0 = fmaf(-q, fmaf(e0.x, yg, ((2.f * e0.y) * yg) * yg), f0.y * yg);
                    const float h1 = fmaf(-q, fmaf(e1.x, yg, ((2.f * e1.y) * yg) * yg), f1.y * yg);
                    const f32x2 H0 = pk2(h0, h0), H1 = pk2(h1, h1);
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        const ulonglong2 z0 = *reinterpret_cast<const ulonglong2*>(tab + 8 * t + 4 * p);
                        const ulonglong2 z1 = *reinterpret_cast<const ulonglong2*>(tab + 8 * u + 4 * p);
                        float a0, a1, b0, b1;
                        upk2(add2(z0.x, H0), a0, a1);
                        upk2(add2(z1.x, H1), b0, b1);
                        s[4 * p] = min3(s[4 * p], a0, b0);
                        s[4 * p + 1] = min3(s[4 * p + 1], a1, b1);
                        upk2(add2(z0.y, H0), a0, a1);
                        upk2(add2(z1.y, H1), b0, b1);
                        s[4 * p + 2] = min3(s[4 * p + 2], a0, b0);
                        s[4 * p + 3] = min3(s[4 * p + 3], a1, b1);
                    }
                }
            }
            // rho: L is convex, so its tangent plane at the centre bounds it from below
#pragma unroll 1
            for (int t = gl; t < k; t += 8) {
                const float4 f = fc[2 * t], e = fc[2 * t + 1];
                const float w2 = 2.f * e.y;
                const float l = fmaf(f.w, dx, fmaf(e.x, dy, fmaf(w2 * dx, dx, fmaf(w2 * dy, dy, 1.f))));
                // (less the rounding of l and its gradient: e.w is 2^-18 of their magnitudes)
                const float r = l - fmaf(fabsf(fmaf(2.f * w2, dx, f.w)), Sx, fmaf(fabsf(fmaf(2.f * w2, dy, e.x)), Sy, e.w));
                rho = fminf(rho, r > 0.f ? r : 0.f);
            }
            // the candidate of the largest bound: the index replaces the low three bits of the bound
            float top = -FLT_MAX;
#pragma unroll
            for (int i = 0; i < 8; i += 2)
                top = max3(top, __uint_as_float((__float_as_uint(s[i]) & ~7u) | i), __uint_as_float((__float_as_uint(s[i + 1]) & ~7u) | (i + 1)));
            all = top;
#pragma unroll
            for (int o = 4; o; o >>= 1) {
                rho = fminf(rho, __shfl_xor_sync(FULL, rho, o));
                all = fmaxf(all, __shfl_xor_sync(FULL, all, o));
            }
            const unsigned own = __ballot_sync(FULL, top == all) & group;
            pj = (__ffs((int)own) - 1) & 7;
            pi = (int)(__float_as_uint(all) & 7u);
        }
        const bool found = k > 0 && all >= 0.f;
        const float cx = fmaf(__shfl_sync(FULL, off, pi), Sx, dx), cy = fmaf(__shfl_sync(FULL, off, pj), Sy, dy);
        float bk = F8<FK>::group_key(co, k, cx, cy, lane);
        if (level < 0) {
            qOld = qLast = bk;
            continue;
        }
        // order of the candidates: virtual thread, the second of a thread first
        int bo = 2 * (8 * (pi & 3) + pj) + (pi < 4 ? 1 : 0);
        if (!found) { bk = -FLT_MAX; bo = 1 << 30; }
        const float target = fmaxf(bk, qLast);
        cut = below > 0.f ? ((target - (target * 0x1p-14f + 1e-37f)) - q) * (rho * 0.999f) : 0.f;
        if (!(cut > 0.f)) cut = 0.f;
        for (bool again = false;;) {
            unsigned alive = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (!(s[i] < (again ? 0.f : cut))) alive |= 1u << i;
            if (found && gl == pj) alive &= ~(1u << pi);
            if (k <= 0 || all < 0.f) alive = 0;
            if (__any_sync(FULL, alive)) {
                do {
                    const int i = alive ? __ffs((int)alive) - 1 : 0;
                    const float x = fmaf(__shfl_sync(FULL, off, i), Sx, dx);
                    if (alive) {
                        const float key = F8<FK>::key(co, k, x, yg);
                        const int order = 2 * (8 * (i & 3) + gl) + (i < 4 ? 1 : 0);
                        if (key > bk || (key == bk && order < bo)) { bk = key; bo = order; }
                        alive &= alive - 1;
                    }
                } while (__any_sync(FULL, alive));
#pragma unroll
                for (int o = 4; o; o >>= 1) {
                    const float ok = __shfl_xor_sync(FULL, bk, o);
                    const int oo = __shfl_xor_sync(FULL, bo, o);
                    if (ok > bk || (ok == bk && oo < bo)) { bk = ok; bo = oo; }
                }
            }
            // nothing beat the current key: on the last level any candidate above the start's key counts
            const bool more = last && !again && cut > 0.f && !(bk > qOld);
            if (!__any_sync(FULL, more)) break;
            again = true;
        }
        const int vt = bo >> 1, bi = (vt >> 3) + ((bo & 1) ? 0 : 4);
        const float bx = fmaf(__shfl_sync(FULL, off, bi & 7), Sx, dx), by = fmaf(__shfl_sync(FULL, off, vt & 7), Sy, dy);
        if (qLast < bk) { dx = bx; dy = by; qLast = bk; }
        if (last) write = qOld < bk;
        __syncwarp();   // the table is rewritten by the next level
    }
    if (gl == 0 && k > 0 && write) {
        const float pu = bexp2(ex);
        pos[v] = make_float4(c0.x + bscale(dx, pu, ex), c0.y + bscale(dy, pu, ex), c0.z, c0.w);
    }
    __syncwarp();
}

}  // namespace vsdmo
