// mlp_train.cu -- one training step of the proposal network in two launches.
//
// The step as separate GEMM, reduction, Adam and packing launches (mlp.cu) is about thirty launches
// of a few microseconds of work each: 275 us per step of 8,192 rows, of which the tensor cores need
// two. In two launches it takes 29 us of a training call, now bound by the tile kernel's chain of
// dependent phases: 12 us of MMAs and epilogues, 4 us of gathering the rows (behind the update before
// it) and 4 us of writing the gradient partials.
//
//   k_train_tile   one CTA per 128 rows keeps the whole step of its rows in shared memory: gathers the
//                  rows, runs the four layers, the loss gradient, the three data-gradient layers
//                  and, as soon as a layer's operands exist, its weight gradient over the 128 rows
//                  into accumulators of their own in tensor memory. Activations are stored once, in
//                  a layout (element (r, c) at (c / 8) 2048 + (r / 8) 128 + (r % 8) 16 + (c % 8) 2)
//                  whose two strides are uniform, so the same bytes are a K-major operand for
//                  the layers and an MN-major one for the weight gradients: no transposed copies.
//                  Weights stream through three 32 KB buffers, each reloaded as soon as its layer is
//                  done. One more CTA draws the next step's rows.
//   k_train_update sums the CTAs' gradient partials, applies Adam and rewrites the packed BF16 weights;
//                  one more block sums the bias gradients and one the loss.
//
// Every product, rounding and summation order is that of the separate launches: a CTA's weight-gradient
// accumulator is the split-K part of its rows, so parameters are bit for bit the same. Batches whose
// parts are not whole tiles (more than 64 tiles and not a multiple) keep the separate launches.
//
// Rows are drawn like std::uniform_int_distribution over std::mt19937_64 draws them: the 64-bit Mersenne
// twister (Nishimura and Matsumoto) with Lemire's multiply-and-reject ("Fast random integer
// generation in an interval", 2019).
#include "vsdmo_internal.cuh"
#include "mlp.cuh"
#include "tc_gemm.cuh"
#include <cmath>

namespace vsdmo {
namespace mlp {

using tc::pk_off;

namespace {

constexpr unsigned FULL = 0xffffffffu;
// limit of the MMA waits, apart from the load waits' (tc::g_wait_limit_ns) so that a test can make them alone expire
static __device__ unsigned long long g_mma_wait_limit_ns = tc::WAIT_NS;
constexpr int TT = 256;   // threads: warp w takes rows 32 (w & 3) .. + 31, columns 64 (w >> 2) .. + 63
// shared memory (bytes)
constexpr uint32_t S_X = 0, S_H1 = S_X + 24576, S_H2 = S_H1 + 32768, S_H3 = S_H2 + 32768, S_DY = S_H3 + 32768;
constexpr uint32_t S_W0 = S_DY + 4096, S_W1 = S_W0 + 32768, S_W2 = S_W1 + 32768, S_TOTAL = S_W2 + 32768;
constexpr uint32_t S_W4T = S_W0 + 8192;   // second load of buffer 0: W4 (4 x 1 KB), then W4^T (8 KB)
// tensor memory columns
constexpr uint32_t C_ACC = 0, C_DW4 = 128, C_DW1 = 144, C_DW3 = 256, C_DW2 = 384;
// gradient partial of one CTA: matrices with element (r, c) at ((c / 4) 128 + r) 4 + c % 4
constexpr int P_W4 = 0, P_W3 = P_W4 + 128 * OUTP, P_W2 = P_W3 + 128 * HID, P_W1 = P_W2 + 128 * HID;
static_assert(P_W1 + 128 * IN == TRAIN_PART, "partial size");

__device__ __forceinline__ uint32_t u_off(int r, int c) {
    return (uint32_t)(c >> 3) * 2048u + (uint32_t)(r >> 3) * 128u + (uint32_t)(r & 7) * 16u + (uint32_t)(c & 7) * 2u;
}
__device__ __forceinline__ uint64_t desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | ((uint64_t)1 << 46);
}
__device__ __forceinline__ void store8(uint8_t* p, const float* v) {
    __align__(16) __nv_bfloat16 h[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = __float2bfloat16_rn(v[i]);
    *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(h);
}

// D [128 x N] = A . B^T: A an activation tile (K-major), B packed weights (chunks of 32 columns, CHUNK
// bytes apart); issued by one thread
template <int K, int N, uint32_t CHUNK>
__device__ __forceinline__ void layer(uint32_t d, uint32_t a, uint32_t b) {
    const uint64_t da = desc(a, 2048, 128), db = tc::smem_desc(b);
#pragma unroll
    for (int j = 0; j < K / 16; ++j)
        tc::mma_bf16(d, da + (4096u >> 4) * j, db + ((j >> 1) * CHUNK + (j & 1) * 256u) / 16u, tc::idesc_bf16(N), j > 0 ? 1u : 0u);
}
// D [128 x N] (+)= A^T . B over the 128 rows of two activation tiles (both MN-major)
template <int N>
__device__ __forceinline__ void wgrad(uint32_t d, uint32_t a, uint32_t b, bool add) {
    const uint64_t da = desc(a, 128, 2048), db = desc(b, 128, 2048);
#pragma unroll
    for (int j = 0; j < 8; ++j)
        tc::mma_bf16(d, da + 16u * j, db + 16u * j, tc::idesc_bf16(N) | (1u << 15) | (1u << 16), add || j > 0 ? 1u : 0u);
}

// Sum of column `lane` over the warp's 32 rows (v: this row's 32 columns), in the order of the xor-butterfly
// over 16, 8, 4, 2, 1: in every step a lane keeps the half of its columns that its own bit names.
__device__ __forceinline__ float column_sum(float* v, int lane) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const float keep = up ? v[o + i] : v[i], give = up ? v[i] : v[o + i];
            v[i] = keep + __shfl_xor_sync(FULL, give, o);
        }
    }
    return v[0];
}

// ---- rows of a step -----------------------------------------------------------------------------------
constexpr int MT_N = 312, MT_M = 156;

__device__ __forceinline__ unsigned long long mt_next(unsigned long long x0, unsigned long long x1, unsigned long long xm) {
    const unsigned long long x = (x0 & 0xFFFFFFFF80000000ull) | (x1 & 0x7FFFFFFFull);
    return xm ^ (x >> 1) ^ ((x & 1ull) ? 0xB5026F5AA96619E9ull : 0ull);
}
__device__ __forceinline__ unsigned long long mt_temper(unsigned long long x) {
    x ^= (x >> 29) & 0x5555555555555555ull;
    x ^= (x << 17) & 0x71D67FFFEDA60000ull;
    x ^= (x << 37) & 0xFFF7EEE000000000ull;
    return x ^ (x >> 43);
}

// The next `want` rows in [0, n_rows) in the generator's order, by one block. mt_g: 312 state words and the
// place of the next word. Blocks of 312 words are made in two halves (the second needs the first), each
// word tempered and scaled by the thread that made it. A rejected word (one in 2^64 / n_rows) would
// shift all later rows: then one thread makes the whole batch again in order.
__device__ void draw_rows(unsigned long long* __restrict__ mt_g, long n_rows, int want, int* __restrict__ out) {
    __shared__ unsigned long long mt[MT_N + 1];
    const int t = threadIdx.x;
    for (int i = t; i < MT_N; i += TT) mt[i] = mt_g[i];
    const int start = (int)mt_g[MT_N];
    const unsigned long long range = (unsigned long long)n_rows, threshold = (0ull - range) % range;
    __syncthreads();
    bool reject = false;
    auto emit = [&](unsigned long long w, int d) {
        if (d < 0 || d >= want) return;
        const unsigned long long x = mt_temper(w);
        reject |= x * range < threshold;
        out[d] = (int)__umul64hi(x, range);
    };
    for (int i = t; i < MT_N; i += TT)
        if (i >= start) emit(mt[i], i - start);
    int d0 = MT_N - start;   // rows made so far
    for (; d0 < want; d0 += MT_N) {
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            const int i = part * MT_M + t;
            unsigned long long w = 0;
            if (t < MT_M) w = mt_next(mt[i], mt[i + 1 == MT_N ? 0 : i + 1], mt[part ? t : i + MT_M]);
            __syncthreads();
            if (t < MT_M) {
                mt[i] = w;
                emit(w, d0 + i);
            }
            __syncthreads();
        }
    }
    if (__syncthreads_or(reject)) {
        if (t == 0) {
            int pos = start, got = 0;
            for (int i = 0; i < MT_N; ++i) mt[i] = mt_g[i];
            while (got < want) {
                if (pos == MT_N) {
                    for (int i = 0; i < MT_N; ++i)
                        mt[i] = mt_next(mt[i], mt[i + 1 == MT_N ? 0 : i + 1], mt[i < MT_M ? i + MT_M : i - MT_M]);
                    pos = 0;
                }
                const unsigned long long x = mt_temper(mt[pos++]);
                if (x * range >= threshold) out[got++] = (int)__umul64hi(x, range);
            }
            mt[MT_N] = (unsigned long long)pos;
        }
    } else if (t == 0) {
        mt[MT_N] = (unsigned long long)(MT_N - (d0 - want));
    }
    __syncthreads();
    for (int i = t; i <= MT_N; i += TT) mt_g[i] = mt[i];
}

struct TileArgs {
    const float* feats;
    const float* targets;
    const int* idx;          // rows, or null: consecutive
    const uint8_t *W1, *W2, *W3, *W4, *W4T, *W3T, *W2T;
    const float* params;
    float* part;             // [CTAs x TRAIN_PART]
    float *ws4, *ws3, *ws2, *ws1;   // per-warp column sums [B / 32 x columns]
    float* loss_rows;        // [B]
    int* err;
    int B, tiles, ctas;      // rows, tiles per CTA, CTAs with rows
    unsigned long long* mt;  // generator, null: no rows to draw
    int* next;               // next step's rows
    long n_rows;
};

// Programmatic dependent launch: the step's two kernels and the next step's start while the one before
// drains; everything the predecessor writes is read after this wait.
__device__ __forceinline__ void wait_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__global__ void __launch_bounds__(TT, 1) k_train_tile(TileArgs p) {
    extern __shared__ __align__(1024) uint8_t sm[];
    __shared__ __align__(8) uint64_t bars[4];
    __shared__ uint32_t tmem_slot;
    // two flags, each written on one side of a phase's first barrier and read on the other side of its next one: a
    // warp that is late in reading one cannot meet the next phase's write
    __shared__ int s_noload, s_nomma;
    __shared__ __align__(16) float s_bias[3 * HID + 4];
    if ((int)blockIdx.x == p.ctas) {
        // its state was last written by this block of the step before, two launches ago
        wait_predecessor();
        draw_rows(p.mt, p.n_rows, p.B, p.next);
        launch_dependents();
        return;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 64;
    const uint32_t sb = tc::smem_u32(sm);
    uint32_t bar_w[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) bar_w[i] = tc::smem_u32(&bars[i]);
    const uint32_t bar_m = tc::smem_u32(&bars[3]);
    if (tid == 0) {
        for (int i = 0; i < 4; ++i) tc::mbar_init(tc::smem_u32(&bars[i]), 1);
        tc::mbar_init_fence();
        s_noload = s_nomma = 0;
    }
    if (warp == 0) tc::tmem_alloc(tc::smem_u32(&tmem_slot), 512);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    // gradient partial of this CTA's rows: a matrix of `cols` accumulator columns, up to 64 per warp
    auto put = [&](uint32_t col, int base, int cols) {
        float* out = p.part + (size_t)blockIdx.x * TRAIN_PART + base;
#pragma unroll 1
        for (int c = c0; c < min(c0 + 64, cols); c += 16) {
            float v[16];
            tc::tmem_ld16(lane_addr + col + (uint32_t)c, v);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                *reinterpret_cast<float4*>(out + ((size_t)((c >> 2) + k) * 128 + row) * 4) =
                    make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
        }
    };
    const unsigned long long limit = tc::wait_limit(), mma_limit = *(volatile unsigned long long*)&g_mma_wait_limit_ns;
    int loads[3] = { 0, 0, 0 }, seen[3] = { 0, 0, 0 };   // thread 0: loads issued / waited for, per buffer
    uint32_t mphase = 0;
    bool pending = false;
    auto load = [&](int i, uint32_t dst, const uint8_t* src, uint32_t bytes) {
        tc::mbar_expect_tx(bar_w[i], bytes);
        ++loads[i];
        tc::bulk_g2s(sb + dst, src, bytes, bar_w[i]);
    };
    const float scale = 2.f / (3.f * (float)p.B);
    bool stop = false;
    for (int t = 0; t < p.tiles && !stop; ++t) {
        const int tile = blockIdx.x * p.tiles + t;
        if (tid == 0 && t > 0) {
            load(0, S_W0, p.W1, 24576);
            load(1, S_W1, p.W2, 32768);
            load(2, S_W2, p.W3, 32768);
        }
        // rows: thread (r, half) gathers 48 inputs of row r and, for its epilogue row, the targets
        float T3[OUT];
        {
            const int r = tid & 127, half = tid >> 7;   // the first half's r is its epilogue row
            const long src = p.idx ? __ldcg(p.idx + tile * 128 + r) : (long)tile * 128 + r;
            const float* f = p.feats + src * IN + half * 48;
            float4 q[12];
            if ((reinterpret_cast<size_t>(p.feats) & 15) == 0) {
#pragma unroll
                for (int i = 0; i < 12; ++i) q[i] = __ldg(reinterpret_cast<const float4*>(f) + i);
            } else {   // a caller's device array on no 16-byte boundary
#pragma unroll
                for (int i = 0; i < 12; ++i) q[i] = make_float4(__ldg(f + 4 * i), __ldg(f + 4 * i + 1), __ldg(f + 4 * i + 2), __ldg(f + 4 * i + 3));
            }
#pragma unroll
            for (int j = 0; j < OUT; ++j) T3[j] = __ldg(p.targets + src * OUT + j);
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const float v[8] = { q[2 * i].x, q[2 * i].y, q[2 * i].z, q[2 * i].w, q[2 * i + 1].x, q[2 * i + 1].y, q[2 * i + 1].z, q[2 * i + 1].w };
                store8(sm + S_X + u_off(r, 48 * half + 8 * i), v);
            }
        }
        if (t == 0) {
            // the rows do not depend on the step before, the weights do
            wait_predecessor();
            if (tid == 0) {
                load(0, S_W0, p.W1, 24576);
                load(1, S_W1, p.W2, 32768);
                load(2, S_W2, p.W3, 32768);
            }
            for (int i = tid; i < 3 * HID + 4; i += TT) {
                const int off = i < HID ? OFF_B1 + i : i < 2 * HID ? OFF_B2 + i - HID : i < 3 * HID ? OFF_B3 + i - 2 * HID : OFF_B4 + i - 3 * HID;
                s_bias[i] = __ldcg(p.params + off);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc::tc_fence_before();
        __syncthreads();
        // phases: 0-3 the layers, 4-6 the data gradients (with the weight gradient of the layer above), 7 the last weight gradient
        for (int ph = 0; ph < 8; ++ph) {
            if (tid == 0) {
                const int buf = ph == 0 || ph == 3 || ph == 4 ? 0 : ph == 1 || ph == 5 ? 1 : ph == 2 || ph == 6 ? 2 : -1;
                bool ok = true;
                if (buf >= 0 && ph != 4) {
                    ok = tc::mbar_wait_within(bar_w[buf], (uint32_t)(seen[buf] & 1), limit);
                    if (ok) ++seen[buf];
                    else { atomicExch(p.err, tc::TC_TIMEOUT_LOAD); s_noload = 1; }
                }
                if (ok) {
                    tc::tc_fence_after();
                    switch (ph) {
                    case 0: layer<IN, HID, 8192>(tmem + C_ACC, sb + S_X, sb + S_W0); break;
                    case 1: layer<HID, HID, 8192>(tmem + C_ACC, sb + S_H1, sb + S_W1); break;
                    case 2: layer<HID, HID, 8192>(tmem + C_ACC, sb + S_H2, sb + S_W2); break;
                    case 3: layer<HID, OUTP, 1024>(tmem + C_ACC, sb + S_H3, sb + S_W0); break;
                    case 4:
                        layer<OUTP, HID, 8192>(tmem + C_ACC, sb + S_DY, sb + S_W4T);
                        wgrad<OUTP>(tmem + C_DW4, sb + S_H3, sb + S_DY, t > 0);
                        break;
                    case 5:
                        layer<HID, HID, 8192>(tmem + C_ACC, sb + S_H3, sb + S_W1);
                        wgrad<HID>(tmem + C_DW3, sb + S_H3, sb + S_H2, t > 0);
                        break;
                    case 6:
                        layer<HID, HID, 8192>(tmem + C_ACC, sb + S_H2, sb + S_W2);
                        wgrad<HID>(tmem + C_DW2, sb + S_H2, sb + S_H1, t > 0);
                        break;
                    default: wgrad<IN>(tmem + C_DW1, sb + S_H1, sb + S_X, t > 0); break;
                    }
                    tc::mma_commit(bar_m);
                }
            }
            __syncthreads();
            if (s_noload) { stop = true; break; }   // nothing was issued
            pending = true;
            // the epilogues are warp-wide: a warp takes part when the wait of all its lanes succeeded
            if (!__all_sync(FULL, tc::mbar_wait_within(bar_m, mphase, mma_limit))) {
                if (lane == 0) { atomicExch(p.err, tc::TC_TIMEOUT_MMA); s_nomma = 1; }
            } else {
                pending = false;
                mphase ^= 1u;
            }
            tc::tc_fence_after();
            if (!pending && ph < 7) {
                // the buffers whose weights this phase finished with take the next ones
                if (tid == 0) {
                    if (ph == 0) {
                        tc::mbar_expect_tx(bar_w[0], 4 * 1024 + 8192);
                        ++loads[0];
                        for (int c = 0; c < 4; ++c) tc::bulk_g2s(sb + S_W0 + 1024u * c, p.W4 + (size_t)c * 8192, 1024, bar_w[0]);
                        tc::bulk_g2s(sb + S_W4T, p.W4T, 8192, bar_w[0]);
                    } else if (ph == 1) load(1, S_W1, p.W3T, 32768);
                    else if (ph == 2) load(2, S_W2, p.W2T, 32768);
                }
                if (ph < 3) {
                    const float* bias = s_bias + ph * HID + c0;
                    uint8_t* dst = sm + (ph == 0 ? S_H1 : ph == 1 ? S_H2 : S_H3);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float v[32];
                        tc::tmem_ld32(lane_addr + C_ACC + (uint32_t)(c0 + 32 * h), v);
#pragma unroll
                        for (int e = 0; e < 32; e += 4) {
                            const float4 b = *reinterpret_cast<const float4*>(bias + 32 * h + e);
                            v[e] = fmaxf(v[e] + b.x, 0.f); v[e + 1] = fmaxf(v[e + 1] + b.y, 0.f);
                            v[e + 2] = fmaxf(v[e + 2] + b.z, 0.f); v[e + 3] = fmaxf(v[e + 3] + b.w, 0.f);
                        }
#pragma unroll
                        for (int k = 0; k < 4; ++k) store8(dst + u_off(row, c0 + 32 * h + 8 * k), v + 8 * k);
                    }
                } else if (ph == 3) {
                    if (c0 == 0) {
                        float v[16], d[16];
                        tc::tmem_ld16(lane_addr + C_ACC, v);
                        float l = 0.f;
#pragma unroll
                        for (int j = 0; j < OUTP; ++j) {
                            d[j] = 0.f;
                            if (j < OUT) {
                                const float e = (v[j] + s_bias[3 * HID + j]) - T3[j];
                                d[j] = scale * e;
                                l += e * e;
                            }
                        }
                        store8(sm + S_DY + u_off(row, 0), d);
                        store8(sm + S_DY + u_off(row, 8), d + 8);
                        p.loss_rows[tile * 128 + row] = l;
#pragma unroll
                        for (int j = 0; j < OUT; ++j) {
                            float s = __bfloat162float(__float2bfloat16_rn(d[j]));
#pragma unroll
                            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
                            if (lane == 0) p.ws4[(size_t)(tile * 4 + (warp & 3)) * OUTP + j] = s;
                        }
                    }
                } else {
                    // dZ = dH * [H > 0] over the activation it masks
                    uint8_t* buf = sm + (ph == 4 ? S_H3 : ph == 5 ? S_H2 : S_H1);
                    float* ws = (ph == 4 ? p.ws3 : ph == 5 ? p.ws2 : p.ws1) + (size_t)(tile * 4 + (warp & 3)) * HID + c0;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float v[32];
                        tc::tmem_ld32(lane_addr + C_ACC + (uint32_t)(c0 + 32 * h), v);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            uint8_t* q = buf + u_off(row, c0 + 32 * h + 8 * k);
                            const uint4 m = *reinterpret_cast<const uint4*>(q);
                            const __nv_bfloat16* hb = reinterpret_cast<const __nv_bfloat16*>(&m);
#pragma unroll
                            for (int i = 0; i < 8; ++i) v[8 * k + i] = __bfloat162float(hb[i]) > 0.f ? v[8 * k + i] : 0.f;
                            store8(q, v + 8 * k);
                        }
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = __bfloat162float(__float2bfloat16_rn(v[i]));
                        ws[32 * h + lane] = column_sum(v, lane);
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            tc::tc_fence_before();
            __syncthreads();
            if (s_nomma) { stop = true; break; }
        }
    }
    launch_dependents();
    if (!stop) {
        put(C_DW4, P_W4, OUTP);
        put(C_DW3, P_W3, HID);
        put(C_DW2, P_W2, HID);
        put(C_DW1, P_W1, IN);
    }
    // after an expired wait, give copies and MMAs in flight a bounded time to land
    if (tid == 0)
        for (int i = 0; i < 3; ++i)
            for (; seen[i] < loads[i]; ++seen[i]) (void)tc::mbar_wait(bar_w[i], (uint32_t)(seen[i] & 1));
    if (pending) (void)tc::mbar_wait(bar_m, mphase);
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, 512);
    }
}

// ---- update -----------------------------------------------------------------------------------------
constexpr int UT = 256;
constexpr int U_WEIGHT_BLOCKS = TRAIN_PART / UT;
static_assert(TRAIN_PART % UT == 0, "whole blocks of weights");
constexpr int U_BIAS_BLOCKS = 3 * HID / 32 + 1, U_BIAS_ROWS = 256;
struct UpdateArgs {
    float *params, *grads, *m, *v;
    const float* part;
    const float *ws4, *ws3, *ws2, *ws1, *loss_rows;
    uint8_t *W1, *W2, *W3, *W4, *W4T, *W3T, *W2T;
    const float* bias_corr;   // Adam's 1 - beta^step for both moments, null: gradients only
    float* loss;              // sum of the row losses
    const int* err;
    int B, parts;
    float lr;
};

__device__ __forceinline__ void put_bf16(uint8_t* base, size_t off, float w) {
    *reinterpret_cast<__nv_bfloat16*>(base + off) = __float2bfloat16_rn(w);
}

// Adam on parameter i with gradient g; returns the new value
__device__ __forceinline__ float adam(const UpdateArgs& a, int i, float g) {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float mi = b1 * a.m[i] + (1.f - b1) * g;
    const float vi = b2 * a.v[i] + (1.f - b2) * g * g;
    a.m[i] = mi;
    a.v[i] = vi;
    const float w = a.params[i] - a.lr * (mi / a.bias_corr[0]) / (sqrtf(vi / a.bias_corr[1]) + eps);
    a.params[i] = w;
    return w;
}

__global__ void __launch_bounds__(UT) k_train_update(UpdateArgs a) {
    const int b = blockIdx.x, t = threadIdx.x;
    wait_predecessor();
    launch_dependents();
    if (*(volatile const int*)a.err) return;   // an expired wait: the step is not applied
    if (b < U_WEIGHT_BLOCKS) {
        const int e = b * UT + t;
        float g = 0.f;
        const float* q = a.part + e;
        int k = 0;
        for (; k + 32 <= a.parts; k += 32) {
            float x[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = __ldcg(q + (size_t)(k + j) * TRAIN_PART);
#pragma unroll
            for (int j = 0; j < 32; ++j) g += x[j];
        }
        for (; k < a.parts; ++k) g += __ldcg(q + (size_t)k * TRAIN_PART);
        const int base = e < P_W3 ? P_W4 : e < P_W2 ? P_W3 : e < P_W1 ? P_W2 : P_W1;
        const int l = e - base, r = (l >> 2) & 127, c = ((l >> 9) << 2) + (l & 3);
        int i;
        if (base == P_W4) {
            i = OFF_W4 + c * HID + r;
            if (c >= OUT) g = 0.f;   // padded output rows
        } else if (base == P_W3) i = OFF_W3 + r * HID + c;
        else if (base == P_W2) i = OFF_W2 + r * HID + c;
        else i = OFF_W1 + r * IN + c;
        a.grads[i] = g;
        if (!a.bias_corr) return;
        float w = adam(a, i, g);
        if (base == P_W4) {
            if (c >= OUT) { w = 0.f; a.params[i] = 0.f; }
            put_bf16(a.W4, pk_off(c, r, HID), w);
            put_bf16(a.W4T, pk_off(r, c, 32), w);
        } else if (base == P_W3) {
            put_bf16(a.W3, pk_off(r, c, HID), w);
            put_bf16(a.W3T, pk_off(c, r, HID), w);
        } else if (base == P_W2) {
            put_bf16(a.W2, pk_off(r, c, HID), w);
            put_bf16(a.W2T, pk_off(c, r, HID), w);
        } else {
            put_bf16(a.W1, pk_off(r, c, IN), w);
        }
        return;
    }
    if (b < U_WEIGHT_BLOCKS + U_BIAS_BLOCKS) {
        // biases, 32 columns per block: the per-warp column sums, added in row order from shared memory
        __shared__ float col[U_BIAS_ROWS][33];
        const int j0 = (b - U_WEIGHT_BLOCKS) * 32, lyr = j0 / HID;   // the last block holds the 16 of layer 4
        const float* ws = lyr == 0 ? a.ws1 : lyr == 1 ? a.ws2 : lyr == 2 ? a.ws3 : a.ws4;
        const int N = lyr < 3 ? HID : OUTP, c = j0 - lyr * HID + (t & 31), nw = a.B / 32;
        const bool real = lyr < 3 || c < OUT;
        float g = 0.f;
        for (int k0 = 0; k0 < nw; k0 += U_BIAS_ROWS) {
            const int rows = min(U_BIAS_ROWS, nw - k0);
            __syncthreads();
#pragma unroll 16
            for (int k = t >> 5; k < rows; k += UT / 32) col[k][t & 31] = real ? __ldcg(ws + (size_t)(k0 + k) * N + c) : 0.f;
            __syncthreads();
            if (t < 32)
#pragma unroll 8
                for (int k = 0; k < rows; ++k) g += col[k][t];
        }
        if (t < 32 && c < N) {
            const int i = (lyr == 0 ? OFF_B1 : lyr == 1 ? OFF_B2 : lyr == 2 ? OFF_B3 : OFF_B4) + c;
            a.grads[i] = g;
            if (a.bias_corr) {
                adam(a, i, g);
                if (!real) a.params[i] = 0.f;
            }
        }
        return;
    }
    // loss: 256 strided sums and a tree
    __shared__ float sh[UT];
    float s = 0.f;
#pragma unroll 16
    for (int i = t; i < a.B; i += UT) s += __ldcg(a.loss_rows + i);
    sh[t] = s;
    __syncthreads();
    for (int o = UT / 2; o; o >>= 1) {
        if (t < o) sh[t] += sh[t + o];
        __syncthreads();
    }
    if (t == 0) *a.loss = sh[0];
}

}  // namespace

void prepare_train() {
    VSDMO_CUDA(cudaFuncSetAttribute(k_train_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S_TOTAL));
}

// (the limit is a variable of each translation unit that waits)
void set_train_wait_limit(unsigned long long ns) {
    VSDMO_CUDA(cudaMemcpyToSymbol(tc::g_wait_limit_ns, &ns, sizeof(ns)));
    VSDMO_CUDA(cudaMemcpyToSymbol(g_mma_wait_limit_ns, &ns, sizeof(ns)));
}
void set_train_mma_wait_limit(unsigned long long ns) {
    VSDMO_CUDA(cudaDeviceSynchronize());
    VSDMO_CUDA(cudaMemcpyToSymbol(g_mma_wait_limit_ns, &ns, sizeof(ns)));
    VSDMO_CUDA(cudaDeviceSynchronize());
}

int fused_tiles(int B) {
    const int tiles = B / 128, parts = wgrad_parts(B);
    return tiles % parts == 0 ? tiles / parts : 0;
}

namespace {
// launch that may start while its predecessor on the stream drains
template <class Args>
void launch_chained(void (*kernel)(Args), int blocks, int threads, size_t smem, const Args& args, bool chained,
                    cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = chained ? 1 : 0;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    VSDMO_CUDA(cudaLaunchKernelEx(&cfg, kernel, args));
}
}  // namespace

void Model::train_tile(TrainBuffers& w, const float* feats, const float* targets, const int* idx, int B,
                       unsigned long long* mt, int* next, long n_rows, bool rows_only, bool chained, cudaStream_t s) {
    const size_t n = (size_t)(w.rows / 32) * HID;
    TileArgs p{};
    p.feats = feats; p.targets = targets; p.idx = idx;
    p.W1 = W1p.p; p.W2 = W2p.p; p.W3 = W3p.p; p.W4 = W4p.p; p.W4T = W4Tp.p; p.W3T = W3Tp.p; p.W2T = W2Tp.p;
    p.params = params.p;
    p.part = w.part.p;
    p.ws3 = w.ws.p; p.ws2 = w.ws.p + n; p.ws1 = w.ws.p + 2 * n; p.ws4 = w.ws.p + 3 * n;
    p.loss_rows = w.loss_rows.p;
    p.err = err.p;
    p.B = B;
    p.tiles = fused_tiles(B);
    p.ctas = rows_only ? 0 : B / 128 / p.tiles;
    p.mt = mt;
    p.next = next;
    p.n_rows = n_rows;
    // a step reads its rows before it waits for its predecessor, the update before it: they were written by
    // the step before that. The first step's come from the launch just before, so it is not chained.
    launch_chained(k_train_tile, p.ctas + (mt ? 1 : 0), TT, S_TOTAL, p, chained, s);
}

void Model::train_update(TrainBuffers& w, int B, const float* bias_corr, float lr, float* loss, cudaStream_t s) {
    const size_t n = (size_t)(w.rows / 32) * HID;
    UpdateArgs a{};
    a.params = params.p; a.grads = grads.p; a.m = adam_m.p; a.v = adam_v.p;
    a.part = w.part.p;
    a.ws3 = w.ws.p; a.ws2 = w.ws.p + n; a.ws1 = w.ws.p + 2 * n; a.ws4 = w.ws.p + 3 * n;
    a.loss_rows = w.loss_rows.p;
    a.W1 = W1p.p; a.W2 = W2p.p; a.W3 = W3p.p; a.W4 = W4p.p; a.W4T = W4Tp.p; a.W3T = W3Tp.p; a.W2T = W2Tp.p;
    a.bias_corr = bias_corr;
    a.loss = loss;
    a.err = err.p;
    a.B = B;
    a.parts = wgrad_parts(B);
    a.lr = lr;
    launch_chained(k_train_update, U_WEIGHT_BLOCKS + U_BIAS_BLOCKS + 1, UT, 0, a, true, s);
}

void Model::train_fused(TrainBuffers& w, const float* feats, const float* targets, long n_rows, int steps, int B, float lr,
                        uint64_t seed, float* d_hist, cudaStream_t s) {
    w.ensure(B, s);
    // generator state (its seeding recurrence) and Adam's bias corrections of every step
    std::vector<unsigned long long> mt(MT_N + 1);
    mt[0] = seed;
    for (int i = 1; i < MT_N; ++i) mt[i] = 6364136223846793005ull * (mt[i - 1] ^ (mt[i - 1] >> 62)) + (unsigned long long)i;
    mt[MT_N] = MT_N;
    std::vector<float> corr(2 * (size_t)std::max(steps, 1));
    for (int i = 0; i < steps; ++i) {
        corr[2 * i] = 1.f - std::pow(0.9f, (float)(step + 1 + i));
        corr[2 * i + 1] = 1.f - std::pow(0.999f, (float)(step + 1 + i));
    }
    DBuf<unsigned long long> d_mt(mt.size(), s);
    DBuf<float> d_corr(corr.size(), s);
    VSDMO_CUDA(cudaMemcpyAsync(d_mt.p, mt.data(), sizeof(unsigned long long) * mt.size(), cudaMemcpyHostToDevice, s));
    VSDMO_CUDA(cudaMemcpyAsync(d_corr.p, corr.data(), sizeof(float) * corr.size(), cudaMemcpyHostToDevice, s));
    int* rows[2] = { w.idx.p, w.idx.p + w.rows };
    if (steps > 0) train_tile(w, feats, targets, nullptr, B, d_mt.p, rows[0], n_rows, true, false, s);   // the first step's rows
    for (int i = 0; i < steps; ++i) {
        train_tile(w, feats, targets, rows[i & 1], B, i + 1 < steps ? d_mt.p : nullptr, rows[(i + 1) & 1], n_rows, false, i > 0, s);
        train_update(w, B, d_corr.p + 2 * i, lr, d_hist + i, s);
        ++step;
    }
    VSDMO_CUDA(cudaStreamSynchronize(s));   // the host vectors may go
}

void Model::gradients_fused(TrainBuffers& w, const float* feats, const float* targets, int B, cudaStream_t s) {
    w.ensure(B, s);
    train_tile(w, feats, targets, nullptr, B, nullptr, nullptr, 0, false, false, s);
    train_update(w, B, nullptr, 0.f, w.loss.p, s);
}

}  // namespace mlp
}  // namespace vsdmo
