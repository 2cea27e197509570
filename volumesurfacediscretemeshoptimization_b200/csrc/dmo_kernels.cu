// dmo_kernels.cu -- the DMO grid search and the quality reductions.
//
// Grid search (one colour class per launch, one warp per free vertex). Replaces
//   k_optimizeHierarchicalInnerTet<128>  dmo/DMOTetImplCub.h:21-137  (tet interior)
//   k_optimizeHierarchical2DFlat<32>     dmo/DMOTriFlatImplCub.h:24-152 (flat triangles)
// Same search as the reference: N x N (x N) candidates per level centred on the current
// position, half-extent grid_scale * (per-axis max ring distance) shrinking by 2/(N-1) per
// level, the vertex moved to the best candidate (largest ring minimum of the mean ratio,
// lowest linear index x-fastest on ties) when it strictly beats the current position, and
// written back only on improvement. What differs is the arithmetic:
//   * the ring is staged as per-element coefficients in shared memory: relative to the
//     vertex and scaled by an exact power of two, the tet determinant is affine in the
//     candidate p (det = d0 - n.p) and the sum of the six squared edge lengths is
//     quadratic (L = C - 2 s.p + 3|p|^2); the flat-triangle area and edge sum likewise;
//   * the grid is separable: each lane owns 16 (tet) or 2 (2D) candidates; tets are judged by an
//     exact candidate filter first (tet_search.cuh), so few candidates cost a full ring key;
//   * the ring minimum is compared through the monotone transform det^2/L^3 (A/L in 2D),
//     kept as a fraction and compared by cross-multiplication (no cbrt or divide per
//     element); inverted elements key the ring by their most negative det / area, the
//     analogue of the reference returning the negative volume / area;
//   * the block-wide cub::ArgMax becomes a warp reduction on (key, candidate index).
// The library is compiled with --fmad=false: the only fused multiply-adds are the written
// fmaf() calls, so the CPU restatement in oracle/or_dmo.c reproduces every bit.
//
// Quality reductions: k_quality_stats replaces k_updateCurrentQualities + k_findMinimumQuality
// (dmo/DMOTet.cu:45-67) in one deterministic launch; k_quality_histogram and
// k_element_qualities replace k_qualityHistogram / k_getElementQualities (dmo/DMOTet.cu:31-43,69-75).
#include "vsdmo_internal.cuh"
#include "chain.cuh"
#include "tc_gemm.cuh"
#include "angle_metrics.cuh"
#include "tet_search.cuh"
#include "hex_search.cuh"
#include "hex_cond.cuh"
#include "quad_cond.cuh"
#include <cfloat>
#include <cuda_bf16.h>
#include <algorithm>

namespace vsdmo {
namespace {

constexpr unsigned FULL = 0xffffffffu;

// packed position of feature (row, col) in the network's 96-column input operand
__device__ __forceinline__ size_t learned_pk_off(long row, int col) { return tc::pk_off(row, col, 96); }
// launch shape of the tet kernels: one warp per block, so a warp's registers and shared memory go
// to the next vertex as soon as its own is done (searches differ in length by 5 x); one / two / four
// warps per block took 0.404 / 0.437 / 0.443 ms per iteration of the 48^3 cube
constexpr int TET_WARPS = 1;
constexpr int TET_MIN_BLOCKS = 28;   // 72 registers
constexpr int TRI_WARPS = 4;
constexpr int TET_MAX_RING = 512;
constexpr int TRI_MAX_RING = 256;

// (key, index): larger key wins, equal keys -> lower index (cub::ArgMax semantics)
__device__ __forceinline__ void warp_argmax(float& k, int& i) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        float ok = __shfl_xor_sync(FULL, k, o);
        int oi = __shfl_xor_sync(FULL, i, o);
        if (ok > k || (ok == k && oi < i)) { k = ok; i = oi; }
    }
}

// (num, den, det) of tet t at (x, y, z): the operations of tet_key1
__device__ __forceinline__ float tet_piece_key(const float4* __restrict__ co, int t, float x, float y, float z) {
    const float4 c0 = co[2 * t], c1 = co[2 * t + 1];
    const float tx = (3.0f * x) * x, ty = (3.0f * y) * y, tz = (3.0f * z) * z;
    const float det = fmaf(c0.z, z, fmaf(c0.y, y, fmaf(c0.x, x, c0.w)));
    const float L = ((c1.w + fmaf(c1.x, x, tx)) + fmaf(c1.y, y, ty)) + fmaf(c1.z, z, tz);
    return det < 0.f ? det : (det * det) / ((L * L) * L);
}

// a key's order as an unsigned integer, its low 5 bits replaced by the tet index
__device__ __forceinline__ unsigned tet_order_key(float key, int t) {
    const unsigned b = __float_as_uint(key);
    const unsigned o = (b & 0x80000000u) ? ~b : (b | 0x80000000u);   // float order as unsigned order
    return (o & ~31u) | (unsigned)t;
}

// Ring key with the tets spread over the lanes and a warp minimum of the per-tet keys (det if
// negative, else det^2 / L^3): the minimum needs no fixed order, so this costs one tet per lane
// and five shuffles. It can differ from tet_key1 in the last bit when two tets' fractions are
// within rounding of each other, so only the learned search, whose moves are judged by keys of
// this same function, uses it.
__device__ __forceinline__ float tet_key_min(const float4* __restrict__ co, int k, float x, float y, float z, int lane) {
    float m = FLT_MAX;
    for (int t = lane; t < k; t += 32) m = fminf(m, tet_piece_key(co, t, x, y, z));
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fminf(m, __shfl_xor_sync(FULL, m, o));
    return m;
}

// Setup of one tet vertex shared by the plain and the learned search: per-axis extent of the
// ring (DMOTetImplCub.h:54-64), the exact power-of-two scale 2^ex and the element coefficients
// in shared memory. Returns the number of tets, 0 when the vertex is left alone (an empty,
// oversized or degenerate ring). scratch: 512 bytes of shared memory per warp. odd: some tet's L is not
// bounded well above zero on the search box (tet_least), so ring keys depend on the order of the tets (ODD).
//
// Rings of up to 32 tets and 32 vertices come from the ring table: one coalesced row of ring
// vertices and one of 16-bit corner triples per vertex, so every ring position is loaded once
// (14 instead of 72 gathers for a Kuhn vertex) and two dependent loads reach the positions
// instead of three (row pointer, halffaces, positions). Larger rings read their halffaces twice.
template <bool ODD>
__device__ __forceinline__ int tet_setup(const float4* __restrict__ pos, const int* __restrict__ rowptr,
                                         const int4* __restrict__ hf, unsigned corner, int nb, int v, int maxk,
                                         float4 c0, int lane, float grid_scale, float4* co, float4* scratch, float& sx,
                                         float& sy, float& sz, int& ex, bool& odd) {
    odd = false;
    const float4 q = pos[nb];
    const unsigned has = __ballot_sync(FULL, corner != TetRingTable::NONE);
    if (__any_sync(FULL, corner == TetRingTable::LARGE)) {
        float mdx = 0.f, mdy = 0.f, mdz = 0.f;
        const int b = rowptr[v], k = rowptr[v + 1] - b;
        if (k <= 0 || k > maxk) return 0;
        for (int t = lane; t < k; t += 32) {
            const int4 h = hf[b + t];
            const float4 pa = pos[h.x], pb = pos[h.y], pc = pos[h.z];
            mdx = fmaxf(mdx, fmaxf(fabsf(pa.x - c0.x), fmaxf(fabsf(pb.x - c0.x), fabsf(pc.x - c0.x))));
            mdy = fmaxf(mdy, fmaxf(fabsf(pa.y - c0.y), fmaxf(fabsf(pb.y - c0.y), fabsf(pc.y - c0.y))));
            mdz = fmaxf(mdz, fmaxf(fabsf(pa.z - c0.z), fmaxf(fabsf(pb.z - c0.z), fabsf(pc.z - c0.z))));
        }
        mdx = redux_max(mdx); mdy = redux_max(mdy); mdz = redux_max(mdz);
        const float mm = fmaxf(mdx, fmaxf(mdy, mdz));
        if (!(mm > 0.f) || !(mm < FLT_MAX)) return 0;
        (void)frexpf(mm, &ex);
        const float p = exp2_exact(-ex);
        for (int t = lane; t < k; t += 32) {
            const int4 h = hf[b + t];
            const float4 pa = pos[h.x], pb = pos[h.y], pc = pos[h.z];
            const float3 a = make_float3(scale2(pa.x - c0.x, p, -ex), scale2(pa.y - c0.y, p, -ex), scale2(pa.z - c0.z, p, -ex));
            const float3 b3 = make_float3(scale2(pb.x - c0.x, p, -ex), scale2(pb.y - c0.y, p, -ex), scale2(pb.z - c0.z, p, -ex));
            const float3 c = make_float3(scale2(pc.x - c0.x, p, -ex), scale2(pc.y - c0.y, p, -ex), scale2(pc.z - c0.z, p, -ex));
            tet_coeffs(a.x, a.y, a.z, b3.x, b3.y, b3.z, c.x, c.y, c.z, co[2 * t], co[2 * t + 1]);
            if (ODD && !(tet_least(co[2 * t + 1]) > tet_odd_limit(grid_scale)))
                odd |= tet_odd(a, b3, c, grid_scale, scale2(mdx, p, -ex), scale2(mdy, p, -ex), scale2(mdz, p, -ex));
        }
        if (ODD) odd = __any_sync(FULL, odd);
        __syncwarp();
        sx = scale2(mdx, p, -ex); sy = scale2(mdy, p, -ex); sz = scale2(mdz, p, -ex);
        return k;
    }
    const int k = __popc(has);   // the triples fill the row from its start
    const float ux = q.x - c0.x, uy = q.y - c0.y, uz = q.z - c0.z;
    const float mdx = redux_max(fabsf(ux)), mdy = redux_max(fabsf(uy)), mdz = redux_max(fabsf(uz));
    const float mm = fmaxf(mdx, fmaxf(mdy, mdz));
    if (k == 0 || !(mm > 0.f) || !(mm < FLT_MAX)) return 0;
    (void)frexpf(mm, &ex);
    const float p = exp2_exact(-ex);
    scratch[lane] = make_float4(scale2(ux, p, -ex), scale2(uy, p, -ex), scale2(uz, p, -ex), 0.f);
    __syncwarp();
    if (lane < k) {
        const float4 a = scratch[corner & 31u], b = scratch[(corner >> 5) & 31u], c = scratch[corner >> 10];
        float4 K1;
        tet_coeffs(a.x, a.y, a.z, b.x, b.y, b.z, c.x, c.y, c.z, co[2 * lane], K1);
        co[2 * lane + 1] = K1;
        odd = ODD && !(tet_least(K1) > tet_odd_limit(grid_scale));
    }
    sx = scale2(mdx, p, -ex); sy = scale2(mdy, p, -ex); sz = scale2(mdz, p, -ex);
    if (ODD && __any_sync(FULL, odd)) {
        if (odd) {
            const float4 a = scratch[corner & 31u], b = scratch[(corner >> 5) & 31u], c = scratch[corner >> 10];
            odd = tet_odd(make_float3(a.x, a.y, a.z), make_float3(b.x, b.y, b.z), make_float3(c.x, c.y, c.z), grid_scale, sx, sy, sz);
        }
        odd = __any_sync(FULL, odd);
    }
    __syncwarp();
    return k;
}

// position c0 + (dx, dy, dz) 2^ex of a move found in scaled local coordinates
__device__ __forceinline__ float4 tet_unscale(float4 c0, float dx, float dy, float dz, int ex) {
    const float p = exp2_exact(ex);
    return make_float4(c0.x + scale2(dx, p, ex), c0.y + scale2(dy, p, ex), c0.z + scale2(dz, p, ex), c0.w);
}

// Active set (optional, dirty != null): a vertex whose last search found no improvement and
// none of whose ring vertices moved since is skipped -- the search would see the same ring and
// return the same "no move", so skipping changes no result. A search that finds nothing clears
// the vertex's flag; a move sets the flags of its ring vertices (adjacent vertices are never in
// the same colour class, so no flag a launch reads is written by that launch).
__device__ __forceinline__ void tet_mark_ring(const int4* __restrict__ hf, int b, int k, int lane,
                                              uint8_t* __restrict__ dirty) {
    for (int t = lane; t < k; t += 32) {
        const int4 h = hf[b + t];
        dirty[h.x] = 1; dirty[h.y] = 1; dirty[h.z] = 1;
    }
}

__global__ void __launch_bounds__(TET_WARPS * 32, TET_MIN_BLOCKS)
k_dmo_tet(float4* __restrict__ pos, const int* __restrict__ rowptr, const int4* __restrict__ hf,
          TetRingTable ring, int v0, int v1, float grid_scale, int depth, int maxk, uint8_t* __restrict__ dirty,
          unsigned long long* __restrict__ skipped) {
    extern __shared__ float4 smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int v = v0 + blockIdx.x * TET_WARPS + w;
    // the wait's pointer serves the loads only: one that lived through the search would cost two registers
    const size_t row = (size_t)(v - ring.base) * 32 + lane;
    const unsigned corner = ring.corner[row];
    const int nb = ring.nb[row];
    const float4* p = chain_wait(pos);
    if (dirty && !*(volatile uint8_t*)(dirty + v)) {
        if (lane == 0 && skipped) atomicAdd(skipped, 1ull);
        return;
    }
    float4* co = smem + (size_t)w * maxk * 2;
    float* scratch = reinterpret_cast<float*>(smem + (size_t)TET_WARPS * maxk * 2) + w * (TS_WARP_BYTES / 4);
    const float4 c0 = p[v];
    float sx, sy, sz;
    int ex;
    bool odd;
    const int k = tet_setup<true>(p, rowptr, hf, corner, nb, v, maxk, c0, lane, grid_scale, co, reinterpret_cast<float4*>(scratch), sx, sy,
                            sz, ex, odd);
    if (k == 0) return;
    float dx, dy, dz;
    const bool moved = tet_search(co, scratch, k, odd, sx, sy, sz, grid_scale, depth, lane, dx, dy, dz);
    if (moved && lane == 0) pos[v] = tet_unscale(c0, dx, dy, dz, ex);
    if (dirty) {
        if (moved) tet_mark_ring(hf, rowptr[v], k, lane, dirty);
        else if (lane == 0) dirty[v] = 0;
    }
}

// The plain search over a list of vertices of one colour class (the learned mode's fallback):
// warps stride over list[0 .. count[0]). The last warp to finish sets the queue back to empty
// (count[0] = 0; count[1] counts the finished warps), so the next class's learned search
// appends to an empty queue without a separate reset launch.
constexpr int TET_LIST_MIN_BLOCKS = 24;   // 80 registers
__global__ void __launch_bounds__(TET_WARPS * 32, TET_LIST_MIN_BLOCKS)
k_dmo_tet_list(float4* __restrict__ pos, const int* __restrict__ rowptr, const int4* __restrict__ hf,
               TetRingTable ring, const int* __restrict__ list, int* __restrict__ count, float grid_scale, int depth, int maxk,
               uint8_t* __restrict__ dirty, unsigned long long* __restrict__ moved_count) {
    extern __shared__ float4 smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float4* co = smem + (size_t)w * maxk * 2;
    float* scratch = reinterpret_cast<float*>(smem + (size_t)TET_WARPS * maxk * 2) + w * (TS_WARP_BYTES / 4);
    const int n = *count;
    for (int idx = blockIdx.x * TET_WARPS + w; idx < n; idx += gridDim.x * TET_WARPS) {
        const int v = list[idx];
        const float4 c0 = pos[v];
        float sx, sy, sz;
        int ex;
        const size_t row = (size_t)(v - ring.base) * 32 + lane;
        bool odd;
        const int k = tet_setup<true>(pos, rowptr, hf, ring.corner[row], ring.nb[row], v, maxk, c0, lane, grid_scale, co,
                                reinterpret_cast<float4*>(scratch), sx, sy, sz, ex, odd);
        if (k == 0) continue;
        float dx, dy, dz;
        const bool moved = tet_search(co, scratch, k, odd, sx, sy, sz, grid_scale, depth, lane, dx, dy, dz);
        if (moved && lane == 0) {
            pos[v] = tet_unscale(c0, dx, dy, dz, ex);
            atomicAdd(moved_count, 1ull);
        }
        if (dirty) {
            if (moved) tet_mark_ring(hf, rowptr[v], k, lane, dirty);
            else if (lane == 0) dirty[v] = 0;
        }
        __syncwarp();
    }
    // every lane of this warp has read count[0]; the last warp of the grid resets the queue (a
    // warp count, not a block barrier: the warps of a block finish their strides apart)
    __syncwarp();
    if (lane == 0) {
        unsigned* done = reinterpret_cast<unsigned*>(count + 1);
        if (atomicAdd(done, 1u) == gridDim.x * TET_WARPS - 1) {
            count[0] = 0;
            *done = 0u;
        }
    }
}

// ---- learned proposal (tet) -------------------------------------------------------------------
// Ring table of the vertices [v0, v1) (the topology is fixed, so it is built once per optimiser):
// the distinct ring vertices of each in first-occurrence order of its halfface row, at most 32
// (nb [(v - v0) * 32 + a], unused places hold v; nbn [v - v0] their number), and the corners of its
// tets as indices into that row (corner [(v - v0) * 32 + t] = a | b << 5 | c << 10, NONE beyond the
// ring; the first is LARGE for a ring of more than 32 tets or vertices). One warp per vertex.
__global__ void __launch_bounds__(128)
k_tet_rings(const int* __restrict__ rowptr, const int4* __restrict__ hf, int v0, int v1, int* __restrict__ nb,
            int* __restrict__ nbn, uint16_t* __restrict__ corner) {
    __shared__ int s_ids[4][96];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int* ids = s_ids[w];
    for (int i = blockIdx.x * 4 + w; i < v1 - v0; i += gridDim.x * 4) {
        const int v = v0 + i;
        const int b = rowptr[v], k = rowptr[v + 1] - b;
        int* out = nb + (size_t)i * 32;
        if (k > 32) {
            int n = 0;
            if (lane == 0) {
                for (int t = 0; t < k; ++t) {
                    const int4 h = hf[b + t];
                    const int u3[3] = { h.x, h.y, h.z };
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        bool seen = false;
                        for (int a = 0; a < n; ++a) seen |= ids[a] == u3[j];
                        if (!seen && n < 32) ids[n++] = u3[j];
                    }
                }
                nbn[i] = n;
            }
            n = __shfl_sync(FULL, n, 0);
            __syncwarp();
            out[lane] = lane < n ? ids[lane] : v;
            corner[(size_t)i * 32 + lane] = TetRingTable::LARGE;
            __syncwarp();
            continue;
        }
        int u3[3] = { v, v, v };
        if (lane < k) {
            const int4 h = hf[b + lane];
            u3[0] = h.x; u3[1] = h.y; u3[2] = h.z;
            ids[3 * lane] = h.x; ids[3 * lane + 1] = h.y; ids[3 * lane + 2] = h.z;
        }
        __syncwarp();
        // place of the first occurrence of each corner among the 3 k corners
        int f3[3] = { 96, 96, 96 };
        for (int q = 3 * k - 1; q >= 0; --q) {
            const int u = ids[q];
#pragma unroll
            for (int j = 0; j < 3; ++j)
                if (u == u3[j]) f3[j] = q;
        }
        unsigned first[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) first[j] = __ballot_sync(FULL, lane < k && f3[j] == 3 * lane + j);
        const int n = __popc(first[0]) + __popc(first[1]) + __popc(first[2]);
        unsigned code = 0;
        int r3[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int tt = min(f3[j] / 3, 31), jj = f3[j] - 3 * (f3[j] / 3);
            const unsigned lower = (1u << tt) - 1u;
            int r = __popc(first[0] & lower) + __popc(first[1] & lower) + __popc(first[2] & lower);
            if (jj > 0) r += (first[0] >> tt) & 1u;
            if (jj > 1) r += (first[1] >> tt) & 1u;
            r3[j] = r;
            code |= (unsigned)(r & 31) << (5 * j);
        }
        __syncwarp();
        if (lane >= n) out[lane] = v;
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (((first[j] >> lane) & 1u) && r3[j] < 32) out[r3[j]] = u3[j];
        if (lane == 0) nbn[i] = min(n, 32);
        corner[(size_t)i * 32 + lane] = n > 32 ? TetRingTable::LARGE : lane < k ? (uint16_t)code : TetRingTable::NONE;
        __syncwarp();
    }
}

// Features of the vertices [v0, v1): the ring vertices nb (in first-occurrence order of the
// halfface row, at most 32) relative to the vertex and divided by the ring's largest
// per-axis extent mm, zero padded to 96 values; FP32 rows and / or BF16 packed rows of the
// network's input operand. scale[i] = mm, old[i] = the vertex position. nb / nbn index the
// range relative to nb_base (the first vertex of the table).
__global__ void k_tet_features(const float4* __restrict__ pos, int v0, int v1, const int* __restrict__ nb,
                               const int* __restrict__ nbn, int nb_base, float* __restrict__ feats,
                               uint8_t* __restrict__ packed, float* __restrict__ scale, float4* __restrict__ old) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < v1 - v0; i += gridDim.x * blockDim.x) {
        const int v = v0 + i;
        const float4 c0 = pos[v];
        const int* list = nb + (size_t)(v - nb_base) * 32;
        const int n = nbn[v - nb_base];
        // each ring vertex loaded once; the 96 inputs stay in registers (fully unrolled)
        float f[96];
        float mm = 0.f;
#pragma unroll
        for (int a = 0; a < 32; ++a) {
            float dx = 0.f, dy = 0.f, dz = 0.f;
            if (a < n) {
                const float4 q = pos[list[a]];
                dx = q.x - c0.x; dy = q.y - c0.y; dz = q.z - c0.z;
                mm = fmaxf(mm, fmaxf(fabsf(dx), fmaxf(fabsf(dy), fabsf(dz))));
            }
            f[3 * a] = dx; f[3 * a + 1] = dy; f[3 * a + 2] = dz;
        }
        const float inv = mm > 0.f ? 1.f / mm : 0.f;
#pragma unroll
        for (int c = 0; c < 96; ++c) f[c] = f[c] * inv;
        if (scale) scale[i] = mm;
        if (old) old[i] = c0;
        if (feats) {
            float4* o = reinterpret_cast<float4*>(feats + (size_t)i * 96);
#pragma unroll
            for (int g = 0; g < 24; ++g) o[g] = make_float4(f[4 * g], f[4 * g + 1], f[4 * g + 2], f[4 * g + 3]);
        }
        if (packed) {
#pragma unroll
            for (int g = 0; g < 12; ++g) {
                __align__(16) __nv_bfloat16 h[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) h[e] = __float2bfloat16_rn(f[8 * g + e]);
                *reinterpret_cast<uint4*>(packed + learned_pk_off(i, 8 * g)) = *reinterpret_cast<const uint4*>(h);
            }
        }
    }
}

// training targets of the vertices [v0, v1) after a plain colour launch: the displacement the
// search chose, in units of the ring extent
__global__ void k_tet_targets(const float4* __restrict__ pos, int v0, int v1, const float* __restrict__ scale,
                              const float4* __restrict__ old, float* __restrict__ targets) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < v1 - v0; i += gridDim.x * blockDim.x) {
        const float4 p = pos[v0 + i], o = old[i];
        const float inv = scale[i] > 0.f ? 1.f / scale[i] : 0.f;
        targets[(size_t)i * 3 + 0] = (p.x - o.x) * inv;
        targets[(size_t)i * 3 + 1] = (p.y - o.y) * inv;
        targets[(size_t)i * 3 + 2] = (p.z - o.z) * inv;
    }
}

// offsets of the reduced grid with n points per axis: (n - 1 - 2i) / (n - 1)
// The 4^3 reduced search ranks its candidates by the LEARNED_CRIT tets of smallest exact key
// at the level's centre (ties to the lower tet), then judges the best-ranked one by its full
// ring key: within the small grid around the proposal the ring minimum of a candidate almost
// always sits in one of those tets, and a third of the ring costs a third of the search.
constexpr int LEARNED_CRIT = 8;

__device__ __forceinline__ void learned_critical(const float4* __restrict__ co, int k, float x, float y, float z,
                                                 int lane, int (&crit)[LEARNED_CRIT]) {
    if (k <= 32) {
        unsigned mine = lane < k ? tet_order_key(tet_piece_key(co, lane, x, y, z), lane) : 0xffffffffu;
#pragma unroll
        for (int r = 0; r < LEARNED_CRIT; ++r) {
            const unsigned m = __reduce_min_sync(FULL, mine);
            const int t = (int)(m & 31u);
            crit[r] = t < k ? t : 0;
            if (lane == t) mine = 0xffffffffu;
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < LEARNED_CRIT; ++r) {
        unsigned best = 0xffffffffu;
        int bt = 0;
        for (int t = lane; t < k; t += 32) {
            bool used = false;
#pragma unroll
            for (int q = 0; q < r; ++q) used |= (crit[q] == t);
            if (used) continue;
            const unsigned kt = tet_order_key(tet_piece_key(co, t, x, y, z), t & 31);
            if (kt < best || (kt == best && t < bt)) { best = kt; bt = t; }
        }
        const unsigned m = __reduce_min_sync(FULL, best);
        const unsigned tt = __reduce_min_sync(FULL, best == m ? (unsigned)bt : 0xffffffffu);
        crit[r] = tt < (unsigned)k ? (int)tt : 0;
    }
}

__device__ __forceinline__ float reduced_offset(int i, int n) { return (float)(n - 1 - 2 * i) / (float)(n - 1); }

// Learned search: the network's displacement y (units of mm) centres a reduced grid of
// rn^3 candidates per level, rdepth levels, half-extent starting at the plain search's second
// level (grid_scale * 2/7 of the ring extent) and shrinking by 2/(rn-1); the proposal itself is
// a candidate too. The vertex moves when the best of them strictly raises its ring minimum;
// otherwise the full plain search runs (fallback), so every move is one plain DMO could
// accept and the minimum quality never decreases. counters: [0] reduced accepted,
// [1] fallbacks, [2] fallbacks that moved, [3] skipped by the active set. rscale: first
// reduced half-extent in units of grid_scale x the per-axis ring extent.
constexpr int TET_LEARNED_MIN_BLOCKS = 32;   // 64 registers (32 bytes of spills): 32 warps per SM
__global__ void __launch_bounds__(TET_WARPS * 32, TET_LEARNED_MIN_BLOCKS)
k_dmo_tet_learned(float4* __restrict__ pos, const int* __restrict__ rowptr, const int4* __restrict__ hf,
                  TetRingTable ring, int v0, int v1, float grid_scale, int maxk, const float* __restrict__ Y, int ldy, int rn, int rdepth,
                  float rscale, unsigned long long* __restrict__ counters, uint8_t* __restrict__ dirty,
                  int* __restrict__ fb_list, int* __restrict__ fb_count) {
    extern __shared__ float4 smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int v = v0 + blockIdx.x * TET_WARPS + w;
    if (v >= v1) return;
    if (dirty && !dirty[v]) {
        if (lane == 0) atomicAdd(&counters[3], 1ull);
        return;
    }
    float4* co = smem + (size_t)w * maxk * 2;
    const float4 c0 = pos[v];
    float sx, sy, sz;
    int ex;
    float4* scratch = smem + (size_t)TET_WARPS * maxk * 2 + w * 32;
    const size_t row = (size_t)(v - ring.base) * 32 + lane;
    bool odd;   // unused: keys here are a minimum over the tets
    const int k = tet_setup<false>(pos, rowptr, hf, ring.corner[row], ring.nb[row], v, maxk, c0, lane, grid_scale, co, scratch, sx, sy, sz, ex, odd);
    if (k == 0) return;
    const float q0 = tet_key_min(co, k, 0.f, 0.f, 0.f, lane);
    // proposal in scaled local coordinates (the features were divided by mm = max(sx, sy, sz) 2^ex)
    const float mms = fmaxf(sx, fmaxf(sy, sz));
    const float* y = Y + (size_t)(v - v0) * ldy;
    float px = y[0] * mms, py = y[1] * mms, pz = y[2] * mms;
    const float bx = grid_scale * sx, by = grid_scale * sy, bz = grid_scale * sz;
    const bool have = isfinite(px) && isfinite(py) && isfinite(pz);
    float best = -FLT_MAX, cx = 0.f, cy = 0.f, cz = 0.f;
    if (have) {
        px = fminf(fmaxf(px, -bx), bx); py = fminf(fmaxf(py, -by), by); pz = fminf(fmaxf(pz, -bz), bz);
        best = tet_key_min(co, k, px, py, pz, lane);
        cx = px; cy = py; cz = pz;
        float rx = grid_scale * rscale * sx, ry = grid_scale * rscale * sy, rz = grid_scale * rscale * sz;
        const int nc = rn * rn * rn;
        for (int level = 0; level < rdepth; ++level) {
            float bk = -FLT_MAX;
            int bi = 1 << 30;
            if (rn == 4) {
                // 64 candidates, index ix + 4 iy + 16 iz: lane (ix, iy, iz0) also takes iz0 + 2,
                // sharing the x and y parts of every tet; offsets (3 - 2i) / 3; ranked over the
                // critical tets of the centre
                const int ix = lane & 3, iy = (lane >> 2) & 3, iz0 = lane >> 4;
                const float o4[4] = { 1.0f, 1.0f / 3.0f, -1.0f / 3.0f, -1.0f };
                const float x = fmaf(o4[ix], rx, cx);
                const float yy = fmaf(o4[iy], ry, cy);
                const float z0 = fmaf(o4[iz0], rz, cz), z1 = fmaf(o4[iz0 + 2], rz, cz);
                const float tx = (3.0f * x) * x, ty = (3.0f * yy) * yy;
                const float tz0 = (3.0f * z0) * z0, tz1 = (3.0f * z1) * z1;
                float N0 = 0.f, D0 = 1.f, m0 = 0.f, N1 = 0.f, D1 = 1.f, m1 = 0.f;
                int crit[LEARNED_CRIT];
                learned_critical(co, k, cx, cy, cz, lane, crit);
                const int nt = min(LEARNED_CRIT, k);
#pragma unroll
                for (int r = 0; r < LEARNED_CRIT; ++r) {
                    if (r >= nt) break;
                    const int t = crit[r];
                    const float4 K0 = co[2 * t], K1 = co[2 * t + 1];
                    const float detB = fmaf(K0.y, yy, fmaf(K0.x, x, K0.w));
                    const float LB = (K1.w + fmaf(K1.x, x, tx)) + fmaf(K1.y, yy, ty);
                    const float d0 = fmaf(K0.z, z0, detB), L0 = LB + fmaf(K1.z, z0, tz0);
                    const float d1 = fmaf(K0.z, z1, detB), L1 = LB + fmaf(K1.z, z1, tz1);
                    const float n0 = d0 * d0, e0 = (L0 * L0) * L0, n1 = d1 * d1, e1 = (L1 * L1) * L1;
                    if (r == 0) { N0 = n0; D0 = e0; m0 = d0; N1 = n1; D1 = e1; m1 = d1; continue; }
                    if (n0 * D0 < N0 * e0) { N0 = n0; D0 = e0; }
                    if (n1 * D1 < N1 * e1) { N1 = n1; D1 = e1; }
                    m0 = fminf(m0, d0); m1 = fminf(m1, d1);
                }
                const float k0 = m0 < 0.f ? m0 : N0 / D0, k1 = m1 < 0.f ? m1 : N1 / D1;
                bk = k0; bi = lane;
                if (k1 > bk) { bk = k1; bi = lane + 32; }
            } else {
                for (int c = lane; c < nc; c += 32) {
                    const int ix = c % rn, iy = (c / rn) % rn, iz = c / (rn * rn);
                    const float x = fmaf(reduced_offset(ix, rn), rx, cx);
                    const float yy = fmaf(reduced_offset(iy, rn), ry, cy);
                    const float z = fmaf(reduced_offset(iz, rn), rz, cz);
                    const float key = tet_key1(co, k, x, yy, z);
                    if (key > bk || (key == bk && c < bi)) { bk = key; bi = c; }
                }
            }
            warp_argmax(bk, bi);
            if (rn == 4 && bi < nc && bk > best) {
                // the best-ranked candidate is judged by its full ring key
                const int ix = bi % rn, iy = (bi / rn) % rn, iz = bi / (rn * rn);
                bk = tet_key_min(co, k, fmaf(reduced_offset(ix, rn), rx, cx), fmaf(reduced_offset(iy, rn), ry, cy),
                                 fmaf(reduced_offset(iz, rn), rz, cz), lane);
            }
            if (bi < nc && bk > best) {
                const int ix = bi % rn, iy = (bi / rn) % rn, iz = bi / (rn * rn);
                const float nx = fmaf(reduced_offset(ix, rn), rx, cx);
                const float ny = fmaf(reduced_offset(iy, rn), ry, cy);
                const float nz = fmaf(reduced_offset(iz, rn), rz, cz);
                cx = nx; cy = ny; cz = nz;
                best = bk;
            }
            const float sh = 2.0f / (float)(rn - 1);
            rx *= sh; ry *= sh; rz *= sh;
        }
    }
    if (have && best > q0) {
        if (lane == 0) {
            pos[v] = tet_unscale(c0, cx, cy, cz, ex);
            atomicAdd(&counters[0], 1ull);
        }
        if (dirty) tet_mark_ring(hf, rowptr[v], k, lane, dirty);
        return;
    }
    // the proposal did not raise the ring minimum: queue the vertex for the plain search
    if (lane == 0) {
        fb_list[atomicAdd(fb_count, 1)] = v;
        atomicAdd(&counters[1], 1ull);
    }
}


// ---- hexahedra ------------------------------------------------------------------------------------
// k_optimizeHierarchicalInnerHex<128> (dmo/DMOHexImplCub.h:21-137) with shapeMetricHex
// (dmo/DMOQualityHex.h:54-71): one warp per vertex stages the halfhexes' coefficients (hex_key.cuh)
// and runs the filtered search of hex_search.cuh. A block of 128 threads that judged all 512
// candidates by the whole ring took 2.14 ms per iteration of the 32^3 cube (10 iterations), this one
// takes 0.50 ms: 17 colour classes of up to 2,600 vertices, one wave each, bound by one search's latency.
constexpr int HEX_MAX_RING = 64;
constexpr int HEX_MIN_BLOCKS = 20;   // 96 registers
// Classes of up to so many vertices (one wave of five blocks per SM) get four warps per vertex, for the levels that are
// evaluated in full: a lattice of 12^3 cells with 1e-6 of jitter takes 441 us per iteration, 868 with one warp (554 with
// every candidate in a block of 128 threads, as before the filter).
constexpr int HEX_TEAM_MAX = 148 * (HEX_MIN_BLOCKS / 4);

// coefficients, then the corners of the setup or the search's scratch and item list
size_t hex_smem_bytes(int maxk) {
    return (size_t)maxk * HEX_CO * sizeof(float) +
           std::max((size_t)TS_WARP_BYTES + 6 * maxk * sizeof(unsigned short), (size_t)7 * maxk * sizeof(float4));
}

template <int W>
__device__ __forceinline__ void hex_vertex(float4* __restrict__ pos, const int* __restrict__ rowptr, const int4* __restrict__ hh, int v,
                                           float grid_scale, int depth, int maxk, float4* smem, HexTeam* team) {
    const int lane = threadIdx.x & 31;
    float* co = reinterpret_cast<float*>(smem);
    float4* corner = smem + maxk * (HEX_CO / 4);
    const int b = rowptr[v], k = rowptr[v + 1] - b;
    if (k <= 0 || k > maxk) return;
    const float4 c0 = pos[v];
    // per-axis largest (scale) and smallest (grid extent, DMOHexImplCub.h:49-68) ring distance
    float mx0 = 0.f, mx1 = 0.f, mx2 = 0.f, mn0 = FLT_MAX, mn1 = FLT_MAX, mn2 = FLT_MAX;
    for (int idx = lane; idx < 7 * k; idx += 32) {
        const int h = idx / 7, c = idx % 7;
        const int4 q = hh[2 * (b + h) + (c >> 2)];
        const int cc = c & 3;
        const float4 p = pos[cc == 0 ? q.x : (cc == 1 ? q.y : (cc == 2 ? q.z : q.w))];
        const float4 d = make_float4(p.x - c0.x, p.y - c0.y, p.z - c0.z, 0.f);
        corner[idx] = d;
        mx0 = fmaxf(mx0, fabsf(d.x)); mx1 = fmaxf(mx1, fabsf(d.y)); mx2 = fmaxf(mx2, fabsf(d.z));
        mn0 = fminf(mn0, fabsf(d.x)); mn1 = fminf(mn1, fabsf(d.y)); mn2 = fminf(mn2, fabsf(d.z));
    }
    mx0 = redux_max(mx0); mx1 = redux_max(mx1); mx2 = redux_max(mx2);
    mn0 = redux_min(mn0); mn1 = redux_min(mn1); mn2 = redux_min(mn2);
    const float mm = fmaxf(mx0, fmaxf(mx1, mx2));
    if (!(mm > 0.f) || !(mm < FLT_MAX)) return;
    int ex;
    (void)frexpf(mm, &ex);
    const float p2 = exp2_exact(-ex);
    const float es = ldexpf(HEX_EPS, -3 * ex), ea = ldexpf(HEX_EPS, -2 * ex);
    const float sx = scale2(mn0, p2, -ex), sy = scale2(mn1, p2, -ex), sz = scale2(mn2, p2, -ex);
    const float X = (1.5f * grid_scale) * sx, Y = (1.5f * grid_scale) * sy, Z = (1.5f * grid_scale) * sz;
    bool odd = false;
    __syncwarp();
    for (int h = lane; h < k; h += 32) {
        float r[7][3];
#pragma unroll
        for (int c = 0; c < 7; ++c) {
            const float4 d = corner[7 * h + c];
            r[c][0] = scale2(d.x, p2, -ex); r[c][1] = scale2(d.y, p2, -ex); r[c][2] = scale2(d.z, p2, -ex);
        }
        hex_coeffs(r, es, ea, co + HEX_CO * h);
        odd |= hex_odd(co + HEX_CO * h, X, Y, Z);
    }
    __syncwarp();
    const HexItems ring{co, k, es, ea, nullptr, 0};
    float* scratch = reinterpret_cast<float*>(corner);
    float dx, dy, dz;
    const bool moved = hex_plain_search<W>(ring, __any_sync(FULL, odd), team, scratch, reinterpret_cast<unsigned short*>(scratch + TS_WARP_BYTES / 4),
                                        sx, sy, sz, grid_scale, depth, lane, dx, dy, dz);
    if (moved && lane == 0) pos[v] = tet_unscale(c0, dx, dy, dz, ex);
}

template <int W>
__global__ void __launch_bounds__(32 * W, W == 1 ? HEX_MIN_BLOCKS : HEX_MIN_BLOCKS / W)
k_dmo_hex(float4* __restrict__ pos, const int* __restrict__ rowptr, const int4* __restrict__ hh, int v0,
          float grid_scale, int depth, int maxk) {
    extern __shared__ float4 smem[];
    const int v = v0 + blockIdx.x;
    if (W == 1) {
        hex_vertex<1>(pos, rowptr, hh, v, grid_scale, depth, maxk, smem, nullptr);
        return;
    }
    __shared__ HexTeam team;
    const int w = threadIdx.x >> 5;
    if (w > 0) {
        hex_team_help(&team, reinterpret_cast<float*>(smem), w);
        return;
    }
    hex_vertex<W>(pos, rowptr, hh, v, grid_scale, depth, maxk, smem, &team);
    if ((threadIdx.x & 31) == 0) team.go = 0;
    __syncthreads();
}

// ---- flat triangles ---------------------------------------------------------------------------
__device__ __forceinline__ float tri_key(const float4* co, int k, float x, float y) {
    const float tx = (2.0f * x) * x, ty = (2.0f * y) * y;
    float N = 0.f, D = 1.f, am = 0.f;
    for (int t = 0; t < k; ++t) {
        const float4 c0 = co[2 * t], c1 = co[2 * t + 1];
        const float A = fmaf(c0.y, y, fmaf(c0.x, x, c0.z));
        const float L = (c0.w + fmaf(c1.x, x, tx)) + fmaf(c1.y, y, ty);
        if (t == 0) { N = A; D = L; am = A; continue; }
        if (A * D < N * L) { N = A; D = L; }
        am = fminf(am, A);
    }
    return am < 0.f ? am : N / D;
}

// tri_key of (x1, y) and (x2, y): one pass over the ring, the two folds' chains side by side
__device__ __forceinline__ void tri_key2(const float4* co, int k, float x1, float x2, float y, float& q1, float& q2) {
    const float t1 = (2.0f * x1) * x1, t2 = (2.0f * x2) * x2, ty = (2.0f * y) * y;
    float N1 = 0.f, D1 = 1.f, a1 = 0.f, N2 = 0.f, D2 = 1.f, a2 = 0.f;
    for (int t = 0; t < k; ++t) {
        const float4 c0 = co[2 * t], c1 = co[2 * t + 1];
        const float A1 = fmaf(c0.y, y, fmaf(c0.x, x1, c0.z)), A2 = fmaf(c0.y, y, fmaf(c0.x, x2, c0.z));
        const float L1 = (c0.w + fmaf(c1.x, x1, t1)) + fmaf(c1.y, y, ty), L2 = (c0.w + fmaf(c1.x, x2, t2)) + fmaf(c1.y, y, ty);
        if (t == 0 || A1 * D1 < N1 * L1) { N1 = A1; D1 = L1; }
        if (t == 0 || A2 * D2 < N2 * L2) { N2 = A2; D2 = L2; }
        a1 = t == 0 ? A1 : fminf(a1, A1);
        a2 = t == 0 ? A2 : fminf(a2, A2);
    }
    q1 = a1 < 0.f ? a1 : N1 / D1;
    q2 = a2 < 0.f ? a2 : N2 / D2;
}

// One warp per vertex, a class of a few hundred vertices at a time: bound by the latency of its own chain (topology,
// positions, coefficients, three levels). Chained launches (chain.cuh), the ring read once, both candidates
// of a lane in one pass and the winner by a warp reduction: 44.9 -> 32.2 us per iteration of the 64^2 grid.
__global__ void __launch_bounds__(TRI_WARPS * 32)
k_dmo_tri2d(float4* __restrict__ pos, const int* __restrict__ rowptr, const int4* __restrict__ he,
            int v0, int v1, float grid_scale, int depth, int maxk) {
    extern __shared__ float4 smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int v = v0 + blockIdx.x * TRI_WARPS + w;
    float4* co = smem + (size_t)w * maxk * 2;
    int b = 0, k = 0, first = 0;
    if (v < v1) {
        b = rowptr[v];
        k = rowptr[v + 1] - b;
        if (lane < k) first = he[b + lane].x;
    }
    const float4* src = chain_wait(pos);
    if (k <= 0 || k > maxk) return;
    const float4 c0 = src[v];
    float4 p0 = make_float4(0.f, 0.f, 0.f, 0.f);
    float mdx = 0.f, mdy = 0.f;
    for (int t = lane; t < k; t += 32) {
        const float4 p = src[t == lane ? first : he[b + t].x];
        if (t == lane) p0 = p;
        mdx = fmaxf(mdx, fabsf(p.x - c0.x));
        mdy = fmaxf(mdy, fabsf(p.y - c0.y));
    }
    mdx = redux_max(mdx); mdy = redux_max(mdy);
    const float mm = fmaxf(mdx, mdy);
    if (!(mm > 0.f) || !(mm < FLT_MAX)) return;
    int ex;
    (void)frexpf(mm, &ex);
    const float p = exp2_exact(-ex);
    // rings of up to 32 points lie in the lanes' registers
    const float nx = __shfl_sync(FULL, p0.x, lane + 1 < k ? lane + 1 : 0), ny = __shfl_sync(FULL, p0.y, lane + 1 < k ? lane + 1 : 0);
    for (int t = lane; t < k; t += 32) {
        float4 pa = p0, pb = make_float4(nx, ny, 0.f, 0.f);
        if (k > 32) {
            pa = src[he[b + t].x];
            pb = src[he[b + (t + 1 == k ? 0 : t + 1)].x];
        }
        const float ax = scale2(pa.x - c0.x, p, -ex), ay = scale2(pa.y - c0.y, p, -ex);
        const float bx = scale2(pb.x - c0.x, p, -ex), by = scale2(pb.y - c0.y, p, -ex);
        const float ux = bx - ax, uy = by - ay;
        const float C = ((ax * ax + ay * ay) + (bx * bx + by * by)) + (ux * ux + uy * uy);
        co[2 * t] = make_float4(-uy, ux, ax * uy - ay * ux, C);
        co[2 * t + 1] = make_float4(-2.0f * (ax + bx), -2.0f * (ay + by), 0.f, 0.f);
    }
    __syncwarp();
    const float sx = scale2(mdx, p, -ex), sy = scale2(mdy, p, -ex);
    const int i1 = lane >> 3, j1 = lane & 7;
    const float o1 = grid_offset(i1), o2 = grid_offset(i1 + 4), oj = grid_offset(j1);
    float dx = 0.f, dy = 0.f;
    const float qOld = tri_key(co, k, 0.f, 0.f);
    float qLast = qOld, lastMax = -FLT_MAX;
    float ds = grid_scale;
    for (int level = 0; level < depth; ++level) {
        const float Sx = ds * sx, Sy = ds * sy;
        const float x1 = fmaf(o1, Sx, dx), x2 = fmaf(o2, Sx, dx), y = fmaf(oj, Sy, dy);
        float q1, q2;
        tri_key2(co, k, x1, x2, y, q1, q2);
        float val = q1;
        if (q2 > q1) val = q2;
        const float selx = (q1 > q2) ? x1 : x2;
        float bv = val;
        int bl = lane;
        if (__any_sync(FULL, val != val)) {
            warp_argmax(bv, bl);
        } else {
            bl = __ffs(__ballot_sync(FULL, val == redux_max(val))) - 1;
            bv = __shfl_sync(FULL, val, bl);
        }
        // outside of the branch: with NaN keys the lanes need not agree on bv, and a shuffle waits for all of them
        const float wx = __shfl_sync(FULL, selx, bl), wy = __shfl_sync(FULL, y, bl);
        if (qLast < bv) { dx = wx; dy = wy; qLast = bv; }
        lastMax = bv;
        ds = ds * (2.0f / 7.0f);
    }
    if (qOld < lastMax && lane == 0)
        pos[v] = make_float4(c0.x + scale2(dx, exp2_exact(ex), ex), c0.y + scale2(dy, exp2_exact(ex), ex), c0.z, c0.w);
}

// ---- reference element metrics ---------------------------------------------------------------
// meanRatioMetricTet (dmo/DMOQualityTet.h:119-143)
__device__ __forceinline__ float q_tet(float4 p0, float4 p1, float4 p2, float4 p3) {
    const float e0x = p1.x - p0.x, e0y = p1.y - p0.y, e0z = p1.z - p0.z;
    const float e1x = p2.x - p0.x, e1y = p2.y - p0.y, e1z = p2.z - p0.z;
    const float e2x = p3.x - p0.x, e2y = p3.y - p0.y, e2z = p3.z - p0.z;
    const float cx = e1y * e2z - e1z * e2y, cy = e1z * e2x - e1x * e2z, cz = e1x * e2y - e1y * e2x;
    const float volume = (1.f / 6.f) * ((e0x * cx + e0y * cy) + e0z * cz);
    if (volume < 0.f) return volume;
    const float mu = cbrtf(volume * volume);
    const float e3x = p2.x - p1.x, e3y = p2.y - p1.y, e3z = p2.z - p1.z;
    const float e4x = p3.x - p1.x, e4y = p3.y - p1.y, e4z = p3.z - p1.z;
    const float e5x = p3.x - p2.x, e5y = p3.y - p2.y, e5z = p3.z - p2.z;
    float l = 0.f;
    l += (e0x * e0x + e0y * e0y) + e0z * e0z;
    l += (e1x * e1x + e1y * e1y) + e1z * e1z;
    l += (e2x * e2x + e2y * e2y) + e2z * e2z;
    l += (e3x * e3x + e3y * e3y) + e3z * e3z;
    l += (e4x * e4x + e4y * e4y) + e4z * e4z;
    l += (e5x * e5x + e5y * e5y) + e5z * e5z;
    const float cbrtf9 = 2.0800838230519f;
    return ((12.f * cbrtf9) * mu) / l;
}

// meanRatioMetricTri2D (dmo/DMOQualityTri.h:243-257)
__device__ __forceinline__ float q_tri2d(float4 p0, float4 p1, float4 p2) {
    const float e0x = p1.x - p0.x, e0y = p1.y - p0.y;
    const float e1x = p2.x - p1.x, e1y = p2.y - p1.y;
    const float e2x = p0.x - p2.x, e2y = p0.y - p2.y;
    const float l = ((e0x * e0x + e0y * e0y) + (e1x * e1x + e1y * e1y)) + (e2x * e2x + e2y * e2y);
    const float area = e0x * e1y - e0y * e1x;
    if (area < 0.f) return area;
    return ((2.f * sqrtf(3.f)) * area) / l;
}

// meanRatioMetricTri(p) (dmo/DMOQualityTri.h:260-272), unsigned
__device__ __forceinline__ float q_tri3d(float4 p0, float4 p1, float4 p2) {
    const float e0x = p1.x - p0.x, e0y = p1.y - p0.y, e0z = p1.z - p0.z;
    const float e1x = p2.x - p0.x, e1y = p2.y - p0.y, e1z = p2.z - p0.z;
    const float e2x = p2.x - p1.x, e2y = p2.y - p1.y, e2z = p2.z - p1.z;
    const float l = (((e0x * e0x + e0y * e0y) + e0z * e0z) + ((e1x * e1x + e1y * e1y) + e1z * e1z)) +
                    ((e2x * e2x + e2y * e2y) + e2z * e2z);
    const float cx = e0y * e1z - e0z * e1y, cy = e0z * e1x - e0x * e1z, cz = e0x * e1y - e0y * e1x;
    return ((2.f * sqrtf(3.f)) * sqrtf((cx * cx + cy * cy) + cz * cz)) / l;
}

// meanRatioMetricQuad(p) (dmo/DMOQualityQuad.h:13-28): 2 (A1 + A2) / sum |e|^2
__device__ __forceinline__ float q_quad(float4 p0, float4 p1, float4 p2, float4 p3) {
    const float e0x = p1.x - p0.x, e0y = p1.y - p0.y, e0z = p1.z - p0.z;
    const float e1x = p2.x - p1.x, e1y = p2.y - p1.y, e1z = p2.z - p1.z;
    const float e2x = p3.x - p2.x, e2y = p3.y - p2.y, e2z = p3.z - p2.z;
    const float e3x = p0.x - p3.x, e3y = p0.y - p3.y, e3z = p0.z - p3.z;
    const float l = ((((e0x * e0x + e0y * e0y) + e0z * e0z) + ((e1x * e1x + e1y * e1y) + e1z * e1z)) +
                     ((e2x * e2x + e2y * e2y) + e2z * e2z)) + ((e3x * e3x + e3y * e3y) + e3z * e3z);
    const float m0x = -e0x, m0y = -e0y, m0z = -e0z, m2x = -e2x, m2y = -e2y, m2z = -e2z;
    const float c1x = e1y * m0z - e1z * m0y, c1y = e1z * m0x - e1x * m0z, c1z = e1x * m0y - e1y * m0x;
    const float c2x = e3y * m2z - e3z * m2y, c2y = e3z * m2x - e3x * m2z, c2z = e3x * m2y - e3y * m2x;
    const float a1 = sqrtf((c1x * c1x + c1y * c1y) + c1z * c1z);
    const float a2 = sqrtf((c2x * c2x + c2y * c2y) + c2z * c2z);
    return (2.f * (a1 + a2)) / l;
}

// meanRatioMetricQuad(p, n) with n = +z (dmo/DMOQualityQuad.h:30-50) for flat quads: -1 when a
// corner turns clockwise, else 2 (A1 + A2) / sum |e|^2 (the corner areas are the z components)
__device__ __forceinline__ float q_quad2d(float4 p0, float4 p1, float4 p2, float4 p3) {
    const float e0x = p1.x - p0.x, e0y = p1.y - p0.y, e1x = p2.x - p1.x, e1y = p2.y - p1.y;
    const float e2x = p3.x - p2.x, e2y = p3.y - p2.y, e3x = p0.x - p3.x, e3y = p0.y - p3.y;
    const float l = (((e0x * e0x + e0y * e0y) + (e1x * e1x + e1y * e1y)) + (e2x * e2x + e2y * e2y)) + (e3x * e3x + e3y * e3y);
    const float c1 = e1x * (-e0y) - e1y * (-e0x);
    const float c2 = e3x * (-e2y) - e3y * (-e2x);
    if (c1 < 0.f || c2 < 0.f) return -1.f;
    return (2.f * (c1 + c2)) / l;
}

// shapeMetricHex (dmo/DMOQualityHex.h:54-71) in the reference's operation order, with cbrtf
__device__ float q_hex(const float4* __restrict__ pos, const int* __restrict__ h) {
    float v[8][3];
#pragma unroll
    for (int c = 0; c < 8; ++c) { const float4 p = pos[h[c]]; v[c][0] = p.x; v[c][1] = p.y; v[c][2] = p.z; }
    const float* P[8] = { v[4], v[5], v[6], v[7], v[0], v[1], v[2], v[3] };
    float L[12][3], X[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        L[0][a] = P[1][a] - P[0][a]; L[4][a] = P[4][a] - P[0][a]; L[8][a] = P[5][a] - P[4][a];
        L[1][a] = P[2][a] - P[1][a]; L[5][a] = P[5][a] - P[1][a]; L[9][a] = P[6][a] - P[5][a];
        L[2][a] = P[3][a] - P[2][a]; L[6][a] = P[6][a] - P[2][a]; L[10][a] = P[7][a] - P[6][a];
        L[3][a] = P[3][a] - P[0][a]; L[7][a] = P[7][a] - P[3][a]; L[11][a] = P[7][a] - P[4][a];
        X[0][a] = (((P[1][a] - P[0][a]) + (P[2][a] - P[3][a])) + (P[5][a] - P[4][a])) + (P[6][a] - P[7][a]);
        X[1][a] = (((P[3][a] - P[0][a]) + (P[2][a] - P[1][a])) + (P[7][a] - P[4][a])) + (P[6][a] - P[5][a]);
        X[2][a] = (((P[4][a] - P[0][a]) + (P[5][a] - P[1][a])) + (P[6][a] - P[2][a])) + (P[7][a] - P[3][a]);
    }
    const int T[9][3] = { { 0, 3, 4 }, { 1, 0, 5 }, { 2, 1, 6 }, { 3, 2, 7 }, { 11, 8, 4 },
                          { 8, 9, 5 }, { 9, 10, 6 }, { 10, 11, 7 }, { 0, 1, 2 } };
    const int S[9][3] = { { 1, 1, 1 }, { 1, -1, 1 }, { 1, -1, 1 }, { -1, -1, 1 }, { 1, 1, -1 },
                          { -1, 1, -1 }, { -1, 1, -1 }, { -1, -1, -1 }, { 1, 1, 1 } };
    float ret = 1e30f;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        float e[3][3];
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float val = i == 8 ? X[T[i][j]][a] : L[T[i][j]][a];
                e[j][a] = S[i][j] < 0 ? -val : val;
            }
        float x[3];
        hcross(e[1], e[2], x);
        const float sj = hdot3(e[0], x);
        const float Aj = (hdot3(e[0], e[0]) + hdot3(e[1], e[1])) + hdot3(e[2], e[2]);
        if (sj < HEX_EPS || Aj < HEX_EPS) return 0.f;
        ret = fminf(ret, cbrtf(sj * sj) / Aj);
    }
    return 3.f * ret;
}

__device__ __forceinline__ float element_quality(const int* __restrict__ el, int kind, const float4* __restrict__ pos, long e) {
    if (kind == MK_HEX) return q_hex(pos, el + 8 * e);
    if (kind == MK_HEX_COND) {
        float v[8][3];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float4 p = pos[el[8 * e + c]];
            v[c][0] = p.x; v[c][1] = p.y; v[c][2] = p.z;
        }
        return hc_element_quality(v);
    }
    if (kind == MK_TET_MINA || kind == MK_TET_MAXA) {
        const int4 t = reinterpret_cast<const int4*>(el)[e];
        const float4 a = pos[t.x], b = pos[t.y], c = pos[t.z], d = pos[t.w];
        const float pa[3] = { a.x, a.y, a.z }, pb[3] = { b.x, b.y, b.z }, pc[3] = { c.x, c.y, c.z }, pd[3] = { d.x, d.y, d.z };
        return kind == MK_TET_MINA ? tet_angle<false>(pa, pb, pc, pd) : tet_angle<true>(pa, pb, pc, pd);
    }
    if (kind == MK_TRI2D_MINA || kind == MK_TRI2D_MAXA) {
        const int* t = el + 3 * e;
        const float4 a = pos[t[0]], b = pos[t[1]], c = pos[t[2]];
        return kind == MK_TRI2D_MINA ? tri2d_angle<false>(a.x, a.y, b.x, b.y, c.x, c.y)
                                     : tri2d_angle<true>(a.x, a.y, b.x, b.y, c.x, c.y);
    }
    if (kind == MK_TRI3D_MINA || kind == MK_TRI3D_MAXA) {
        const int* t = el + 3 * e;
        const float4 a = pos[t[0]], b = pos[t[1]], c = pos[t[2]];
        const float pa[3] = { a.x, a.y, a.z }, pb[3] = { b.x, b.y, b.z }, pc[3] = { c.x, c.y, c.z };
        return kind == MK_TRI3D_MINA ? tri3d_angle<false, false>(pa, pb, pc, 0.f, 0.f, 0.f)
                                     : tri3d_angle<true, false>(pa, pb, pc, 0.f, 0.f, 0.f);
    }
    if (kind == MK_TET) {
        const int4 t = reinterpret_cast<const int4*>(el)[e];
        return q_tet(pos[t.x], pos[t.y], pos[t.z], pos[t.w]);
    }
    if (kind == MK_QUAD || kind == MK_QUAD2D) {
        const int4 t = reinterpret_cast<const int4*>(el)[e];
        return kind == MK_QUAD ? q_quad(pos[t.x], pos[t.y], pos[t.z], pos[t.w]) : q_quad2d(pos[t.x], pos[t.y], pos[t.z], pos[t.w]);
    }
    if (kind == MK_QUAD_COND) {
        const int4 t = reinterpret_cast<const int4*>(el)[e];
        const float4 a = pos[t.x];
        return quad_cond<false>(a.x, a.y, a.z, pos[t.y], pos[t.z], pos[t.w], make_float3(0.f, 0.f, 0.f));
    }
    const int* t = el + 3 * e;
    if (kind == MK_TRI3D) return q_tri3d(pos[t[0]], pos[t[1]], pos[t[2]]);
    return q_tri2d(pos[t[0]], pos[t[1]], pos[t[2]]);
}

// the element loop is a chain of dependent loads (indices, then corners), bound by how many of
// them are in flight: four elements per thread, one resident grid (80 registers: 3 blocks of
// 256 threads per SM)
constexpr int QS_BLOCKS = 148 * 3;
constexpr int QS_THREADS = 256;
constexpr int QS_UNROLL = 4;

template <bool CHAINED>
__global__ void __launch_bounds__(QS_THREADS)
k_quality_stats(const int* __restrict__ el, int kind, long nE, const float4* __restrict__ pos_, IterStats* stats,
                int* iter, float* pmin, double* psum, int* pfail, unsigned* done, int check, int init) {
    __shared__ float smin[QS_THREADS / 32];
    __shared__ double ssum[QS_THREADS / 32];
    __shared__ int sfail[QS_THREADS / 32];
    __shared__ bool last;
    const float4* __restrict__ pos = CHAINED ? chain_wait(pos_) : pos_;
    const int it = *iter;
    const float lastMin = init ? -FLT_MAX : stats[it].min_q;
    const float tol = 1e-6f * fmaxf(fabsf(lastMin), 1e-30f);
    float mn = FLT_MAX;
    double sm = 0.0;
    int fl = 0;
    const long st = (long)QS_BLOCKS * QS_THREADS;
    long e = (long)blockIdx.x * QS_THREADS + threadIdx.x;
    for (; e + (QS_UNROLL - 1) * st < nE; e += QS_UNROLL * st) {
        float q[QS_UNROLL];
#pragma unroll
        for (int j = 0; j < QS_UNROLL; ++j) q[j] = element_quality(el, kind, pos, e + j * st);
#pragma unroll
        for (int j = 0; j < QS_UNROLL; ++j) {
            mn = fminf(mn, q[j]);
            sm += (double)q[j];
            if (check && q[j] < lastMin - tol) ++fl;
        }
    }
    for (; e < nE; e += st) {
        const float q = element_quality(el, kind, pos, e);
        mn = fminf(mn, q);
        sm += (double)q;
        if (check && q < lastMin - tol) ++fl;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(FULL, mn, o));
        sm += __shfl_xor_sync(FULL, sm, o);
        fl += __shfl_xor_sync(FULL, fl, o);
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) { smin[w] = mn; ssum[w] = sm; sfail[w] = fl; }
    __syncthreads();
    if (threadIdx.x == 0) {
        float a = smin[0]; double s = ssum[0]; int f = sfail[0];
        for (int i = 1; i < QS_THREADS / 32; ++i) { a = fminf(a, smin[i]); s += ssum[i]; f += sfail[i]; }
        pmin[blockIdx.x] = a; psum[blockIdx.x] = s; pfail[blockIdx.x] = f;
        __threadfence();
        last = atomicAdd(done, 1u) == QS_BLOCKS - 1;
    }
    __syncthreads();
    if (!last) return;
    // the last block folds the partials: thread t takes t, t + QS_THREADS, ... in order, then a
    // fixed tree (the same order every run)
    __threadfence();
    {
        float a = FLT_MAX; double s = 0.0; int f = 0;
        for (int i = threadIdx.x; i < QS_BLOCKS; i += QS_THREADS) {
            a = fminf(a, ((volatile float*)pmin)[i]); s += ((volatile double*)psum)[i]; f += ((volatile int*)pfail)[i];
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            a = fminf(a, __shfl_xor_sync(FULL, a, o));
            s += __shfl_xor_sync(FULL, s, o);
            f += __shfl_xor_sync(FULL, f, o);
        }
        if (lane == 0) { smin[w] = a; ssum[w] = s; sfail[w] = f; }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float a = smin[0]; double s = ssum[0]; int f = sfail[0];
        for (int i = 1; i < QS_THREADS / 32; ++i) { a = fminf(a, smin[i]); s += ssum[i]; f += sfail[i]; }
        const int slot = init ? 0 : it + 1;
        stats[slot].min_q = a;
        stats[slot].sum_q = s;
        stats[slot].fail_count = f;
        if (!init) *iter = it + 1;
        *done = 0u;
    }
}

__global__ void k_element_qualities(const int* __restrict__ el, int kind, long nE, const float4* __restrict__ pos, float* out) {
    for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < nE; e += (long)gridDim.x * blockDim.x)
        out[e] = element_quality(el, kind, pos, e);
}

// Counts per block in shared memory, one copy per warp, and the lanes of a warp that hit the same bin count
// once: a mesh near its optimum has most of its elements in one bin, and adding each of them to global
// memory took 0.9 ms for the 664 k tets of the 48^3 cube. HIST_MAX_BINS bins fit; more count globally.
constexpr int HIST_THREADS = 256;
constexpr int HIST_MAX_BINS = 1024;

__global__ void __launch_bounds__(HIST_THREADS)
k_quality_histogram(const int* __restrict__ el, int kind, long nE, const float4* __restrict__ pos, int* counts, int n_cols) {
    extern __shared__ int hist[];
    const bool local = n_cols <= HIST_MAX_BINS;
    int* mine = hist + (threadIdx.x >> 5) * n_cols;
    if (local) {
        for (int i = threadIdx.x; i < HIST_THREADS / 32 * n_cols; i += HIST_THREADS) hist[i] = 0;
        __syncthreads();
    }
    for (long e0 = (long)blockIdx.x * blockDim.x; e0 < nE; e0 += (long)gridDim.x * blockDim.x) {
        const long e = e0 + threadIdx.x;
        int idx = -1;
        if (e < nE) {
            const float q = fminf(0.9999f, element_quality(el, kind, pos, e));
            idx = q > 0.f ? (int)(q * n_cols) : 0;  // a negative quality lands in bin 0
        }
        const unsigned same = __match_any_sync(FULL, idx);
        if (idx >= 0 && __ffs((int)same) - 1 == (int)(threadIdx.x & 31)) {
            if (local) mine[idx] += __popc(same);   // one lane per bin, the warp's own copy
            else atomicAdd(&counts[idx], __popc(same));
        }
        __syncwarp();
    }
    if (!local) return;
    __syncthreads();
    for (int i = threadIdx.x; i < n_cols; i += HIST_THREADS) {
        int c = 0;
        for (int w = 0; w < HIST_THREADS / 32; ++w) c += hist[w * n_cols + i];
        if (c) atomicAdd(&counts[i], c);
    }
}

}  // namespace

int dmo_tet_max_ring() { return TET_MAX_RING; }
int dmo_hex_max_ring() { return HEX_MAX_RING; }

void launch_dmo_hex(const Mesh& m, const DmoLaunch& L, cudaStream_t s) {
    const int n = L.v1 - L.v0;
    if (n <= 0) return;
    const int maxk = m.maxTets;
    const auto kernel = n <= HEX_TEAM_MAX ? k_dmo_hex<4> : k_dmo_hex<1>;
    kernel<<<n, n <= HEX_TEAM_MAX ? 128 : 32, hex_smem_bytes(maxk), s>>>(m.pos.p, m.hf_rowptr.p, m.hh.p, L.v0, L.grid_scale, L.depth, maxk);
    VSDMO_CHECK_LAUNCH();
}

// coefficients of every warp's ring, then every warp's search scratch
size_t tet_smem_bytes(int maxk) { return (size_t)TET_WARPS * (maxk * 2 * sizeof(float4) + TS_WARP_BYTES); }

// Raises the dynamic shared-memory limit of the grid-search kernels (called once per
// optimiser, outside any stream capture, on the current device).
void prepare_dmo_kernels() {
    VSDMO_CUDA(cudaFuncSetAttribute(k_dmo_tet, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tet_smem_bytes(TET_MAX_RING)));
    VSDMO_CUDA(cudaFuncSetAttribute(k_dmo_tri2d, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    TRI_WARPS * TRI_MAX_RING * 2 * (int)sizeof(float4)));
    VSDMO_CUDA(cudaFuncSetAttribute(k_dmo_tet_learned, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    TET_WARPS * (TET_MAX_RING * 2 + 32) * (int)sizeof(float4)));
    VSDMO_CUDA(cudaFuncSetAttribute(k_dmo_tet_list, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)tet_smem_bytes(TET_MAX_RING)));
    for (auto k : {k_dmo_hex<1>, k_dmo_hex<4>})
        VSDMO_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hex_smem_bytes(HEX_MAX_RING)));
}
int dmo_tri2d_max_ring() { return TRI_MAX_RING; }
int quality_stats_blocks() { return QS_BLOCKS; }

void launch_dmo_tet(const Mesh& m, const DmoLaunch& L, const TetRingTable& ring, cudaStream_t s, uint8_t* dirty,
                    unsigned long long* skipped) {
    const int n = L.v1 - L.v0;
    if (n <= 0) return;
    const int maxk = m.maxTets;
    const size_t smem = tet_smem_bytes(maxk);
    VSDMO_CUDA(launch_chained(k_dmo_tet, (n + TET_WARPS - 1) / TET_WARPS, TET_WARPS * 32, smem, s, L.chained, m.pos.p,
                              m.hf_rowptr.p, m.hf.p, ring, L.v0, L.v1, L.grid_scale, L.depth, maxk, dirty, skipped));
}

// Active set with a free boundary: the boundary passes move vertices whose rings hold interior
// vertices; flagging the rings of all boundary vertices [v0, v1) keeps "skipping changes no
// result" without tracking which boundary vertex moved. One warp per vertex.
__global__ void k_mark_rings(const int* __restrict__ rowptr, const int4* __restrict__ hf, int v0, int v1,
                             uint8_t* __restrict__ dirty) {
    const int v = v0 + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (v >= v1) return;
    const int b = rowptr[v];
    tet_mark_ring(hf, b, rowptr[v + 1] - b, threadIdx.x & 31, dirty);
}

void launch_mark_rings(const Mesh& m, int v0, int v1, uint8_t* dirty, cudaStream_t s) {
    if (v1 <= v0 || !dirty) return;
    const long threads = 32L * (v1 - v0);
    k_mark_rings<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(m.hf_rowptr.p, m.hf.p, v0, v1, dirty);
    VSDMO_CHECK_LAUNCH();
}

void launch_tet_rings(const Mesh& m, int v0, int v1, int* nb, int* nbn, uint16_t* corner, cudaStream_t s) {
    if (v1 <= v0) return;
    k_tet_rings<<<grid_for(32L * (v1 - v0), 128), 128, 0, s>>>(m.hf_rowptr.p, m.hf.p, v0, v1, nb, nbn, corner);
    VSDMO_CHECK_LAUNCH();
}

void launch_tet_features(const Mesh& m, int v0, int v1, const int* nb, const int* nbn, int nb_base, float* feats,
                         uint8_t* packed, float* scale, float4* old, cudaStream_t s) {
    if (v1 <= v0) return;
    k_tet_features<<<grid_for(v1 - v0, 128), 128, 0, s>>>(m.pos.p, v0, v1, nb, nbn, nb_base, feats, packed, scale, old);
    VSDMO_CHECK_LAUNCH();
}

void launch_tet_targets(const Mesh& m, int v0, int v1, const float* scale, const float4* old, float* targets,
                        cudaStream_t s) {
    if (v1 <= v0) return;
    k_tet_targets<<<grid_for(v1 - v0, 256), 256, 0, s>>>(m.pos.p, v0, v1, scale, old, targets);
    VSDMO_CHECK_LAUNCH();
}

void launch_dmo_tet_learned(const Mesh& m, const DmoLaunch& L, const TetRingTable& ring, const float* Y, int ldy,
                            int rn, int rdepth, float rscale, unsigned long long* counters, uint8_t* dirty, int* fb_list, int* fb_count,
                            cudaStream_t s) {
    const int n = L.v1 - L.v0;
    if (n <= 0) return;
    const int maxk = m.maxTets;
    const size_t smem = (size_t)TET_WARPS * (maxk * 2 + 32) * sizeof(float4);
    k_dmo_tet_learned<<<(n + TET_WARPS - 1) / TET_WARPS, TET_WARPS * 32, smem, s>>>(
        m.pos.p, m.hf_rowptr.p, m.hf.p, ring, L.v0, L.v1, L.grid_scale, maxk, Y, ldy, rn, rdepth, rscale, counters, dirty,
        fb_list, fb_count);
    VSDMO_CHECK_LAUNCH();
    // fallback: the plain search over the queued vertices, a fixed grid striding over the list
    const int blocks = std::min((n + TET_WARPS - 1) / TET_WARPS, 148 * TET_LIST_MIN_BLOCKS);
    k_dmo_tet_list<<<blocks, TET_WARPS * 32, tet_smem_bytes(maxk), s>>>(m.pos.p, m.hf_rowptr.p, m.hf.p, ring, fb_list,
                                                                        fb_count, L.grid_scale, L.depth, maxk, dirty, counters + 2);
    VSDMO_CHECK_LAUNCH();
}

void launch_dmo_tri2d(const Mesh& m, const DmoLaunch& L, cudaStream_t s) {
    const int n = L.v1 - L.v0;
    if (n <= 0) return;
    const int maxk = m.maxHE;
    const size_t smem = (size_t)TRI_WARPS * maxk * 2 * sizeof(float4);
    VSDMO_CUDA(launch_chained(k_dmo_tri2d, (n + TRI_WARPS - 1) / TRI_WARPS, TRI_WARPS * 32, smem, s, L.chained, m.pos.p,
                              m.he_rowptr.p, m.he.p, L.v0, L.v1, L.grid_scale, L.depth, maxk));
}

void launch_quality_stats(const Mesh& m, int kind, IterStats* d_stats, int* d_iter, float* d_partial_min,
                          double* d_partial_sum, int* d_partial_fail, unsigned* d_done, int check_monotone,
                          cudaStream_t s, bool chained) {
    // check_monotone < 0 marks the initial evaluation (slot 0, no check, no increment)
    const int init = check_monotone < 0 ? 1 : 0;
    VSDMO_CUDA(launch_chained(chained ? k_quality_stats<true> : k_quality_stats<false>, QS_BLOCKS, QS_THREADS, 0, s, chained, m.elems.p, kind,
                              m.nE, m.pos.p, d_stats, d_iter, d_partial_min, d_partial_sum, d_partial_fail, d_done,
                              init ? 0 : check_monotone, init));
}

void launch_element_qualities(const Mesh& m, int kind, float* d_out, cudaStream_t s) {
    k_element_qualities<<<grid_for(m.nE, 256), 256, 0, s>>>(m.elems.p, kind, m.nE, m.pos.p, d_out);
    VSDMO_CHECK_LAUNCH();
}

void launch_quality_histogram(const Mesh& m, int kind, int* d_counts, int n_cols, cudaStream_t s) {
    const size_t smem = n_cols <= HIST_MAX_BINS ? sizeof(int) * (HIST_THREADS / 32) * n_cols : 0;
    k_quality_histogram<<<grid_for(m.nE, HIST_THREADS, 148 * 4), HIST_THREADS, smem, s>>>(m.elems.p, kind, m.nE, m.pos.p,
                                                                                          d_counts, n_cols);
    VSDMO_CHECK_LAUNCH();
}

}  // namespace vsdmo
