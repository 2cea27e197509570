// prim.cu -- device-wide primitives used by the connectivity build: exclusive scan, stable
// LSD radix sort of (key, value) pairs, stable compaction, rows by key and CSR offsets. These replace the
// thrust::sort_by_key / remove_if / inclusive_scan calls of the reference's mesh build
// (e.g. mesh/MeshTriGPU.cu:142,162-170, mesh/MeshTetGPU.cu:125) and k_find_first_n
// (mesh/SortUtil.cu:3-35). The build runs once per mesh and is bound by launches and latency.
#include "vsdmo_internal.cuh"
#include <mutex>

namespace vsdmo {

namespace {
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;   // per thread
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
constexpr unsigned FULL = 0xffffffffu;

// Prefix sums in two launches: the sums of the tiles, then every block adds up the tile sums before its own
// and scans its tile again (one launch where one tile holds everything). A warp owns 512 consecutive items,
// read 32 at a time. What is summed and where it goes are functors, so that the flags of a
// partition or compaction are read and its indices written by the scan itself. The build is launch-bound: a
// partition was six launches with separate scan levels and flag passes, 13 us against 6 for 117,649 flags.
struct LoadInt {
    const int* a;
    __device__ int operator()(long i) const { return a[i]; }
};
struct LoadFlag {   // flag == first ? 1 : 0
    const uint8_t* f;
    int first;
    __device__ int operator()(long i) const { return ((f[i] != 0) == (first != 0)) ? 1 : 0; }
};
struct StoreInt {
    int* o;
    __device__ void operator()(long i, int before, int, int) const { o[i] = before; }
};
struct StoreFlagged {   // the flagged indices in order
    int* o;
    __device__ void operator()(long i, int before, int v, int) const { if (v) o[before] = (int)i; }
};
struct StorePartition {   // the flagged indices in order, then the others (i - before of them precede i)
    int* o;
    __device__ void operator()(long i, int before, int v, int total) const { o[v ? before : total + (int)(i - before)] = (int)i; }
};

template <class L>
__device__ __forceinline__ int load_tile(L load, long n, int (&v)[SCAN_ITEMS]) {
    const long base = (long)blockIdx.x * SCAN_TILE + (threadIdx.x >> 5) * (32 * SCAN_ITEMS) + (threadIdx.x & 31);
    int s = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
        const long k = base + 32 * i;
        v[i] = k < n ? load(k) : 0;
        s += v[i];
    }
    return __reduce_add_sync(FULL, s);
}

template <class L>
__global__ void __launch_bounds__(SCAN_THREADS) k_tile_sums(L load, long n, int* sums) {
    __shared__ int ws[SCAN_THREADS / 32];
    int v[SCAN_ITEMS];
    const int s = load_tile(load, n, v);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
#pragma unroll
        for (int i = 0; i < SCAN_THREADS / 32; ++i) t += ws[i];
        sums[blockIdx.x] = t;
    }
}

template <class L, class S>
__global__ void __launch_bounds__(SCAN_THREADS) k_tile_scan(L load, S store, long n, const int* sums, int nb, int* total_out) {
    __shared__ int ws[SCAN_THREADS / 32], wb[SCAN_THREADS / 32], wt[SCAN_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int v[SCAN_ITEMS];
    const int s = load_tile(load, n, v);
    int b = 0, t = 0;
    if (nb > 1) {
        for (int i = threadIdx.x; i < nb; i += SCAN_THREADS) {
            const int x = sums[i];
            b += i < (int)blockIdx.x ? x : 0;
            t += x;
        }
        b = __reduce_add_sync(FULL, b);
        t = __reduce_add_sync(FULL, t);
    } else {
        t = s;
    }
    if (lane == 0) { ws[w] = s; wb[w] = b; wt[w] = t; }
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int i = 0; i < SCAN_THREADS / 32; ++i) {
        before += wb[i] + (i < w ? ws[i] : 0);
        total += wt[i];
    }
    if (total_out && blockIdx.x == 0 && threadIdx.x == 0) *total_out = total;
    const long base = (long)blockIdx.x * SCAN_TILE + w * (32 * SCAN_ITEMS) + lane;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
        int x = v[i];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x += y;
        }
        const long k = base + 32 * i;
        if (k < n) store(k, before + x - v[i], v[i], total);
        before += __shfl_sync(FULL, x, 31);
    }
}

template <class L, class S>
void scan(L load, S store, long n, int* total, cudaStream_t s) {
    const long nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    DBuf<int> sums;
    if (nb > 1) {
        sums.alloc(nb, s);
        k_tile_sums<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(load, n, sums.p);
        VSDMO_CHECK_LAUNCH();
    }
    k_tile_scan<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(load, store, n, sums.p, (int)nb, total);
    VSDMO_CHECK_LAUNCH();
}

constexpr int RS_THREADS = 256;
// pairs per tile: 16 per thread, or 4 where that leaves SMs without a tile (148 x 4096 pairs): the sort of
// 103,823 vertices by colour takes 12 us (counts and scatter) against 27
constexpr long RS_SMALL_N = 148L * 4096;
constexpr int RS_WARPS = RS_THREADS / 32;

template <int RS_ROUNDS>
__global__ void k_radix_hist(const uint32_t* keys, long n, int shift, int* counts, int nTiles) {
    __shared__ int h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    constexpr int RS_TILE = RS_THREADS * RS_ROUNDS;
    const long base = (long)blockIdx.x * RS_TILE;
    for (int r = 0; r < RS_ROUNDS; ++r) {
        long idx = base + (long)r * RS_THREADS + threadIdx.x;
        if (idx < n) atomicAdd(&h[(keys[idx] >> shift) & 255u], 1);
    }
    __syncthreads();
    counts[(long)threadIdx.x * nTiles + blockIdx.x] = h[threadIdx.x];
}

// One tile of RS_TILE pairs: the stable rank of every pair within the tile, computed 256 pairs at
// a time (a warp match per digit, warp counts, a running base per digit), places the pair in
// shared memory in tile-local digit order; then consecutive threads write consecutive pairs of
// a digit run to consecutive global positions (the tile's run of digit d starts at its global
// offset offs[d * nTiles + tile]), so the writes coalesce.
template <int RS_ROUNDS>
__global__ void __launch_bounds__(RS_THREADS)
k_radix_scatter(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout, long n, int shift,
                const int* offs, int nTiles) {
    constexpr int RS_TILE = RS_THREADS * RS_ROUNDS;
    __shared__ uint32_t sk[RS_TILE], sv[RS_TILE];
    __shared__ int gbase[256], lstart[256], run[256];
    __shared__ int wcnt[RS_WARPS][257];
    __shared__ int wsum[RS_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const long tile = (long)blockIdx.x * RS_TILE;
    const int tile_n = (int)min((long)RS_TILE, n - tile);
    // the tile's count of digit tid, from the scanned (digit-major) offsets
    const long idx = (long)tid * nTiles + blockIdx.x;
    const int g = offs[idx];
    const int next = (idx + 1 < 256L * nTiles) ? offs[idx + 1] : (int)n;
    const int cnt = next - g;
    gbase[tid] = g;
    // exclusive scan of the counts over the digits: the tile-local run starts
    int x = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    int before = 0;
#pragma unroll
    for (int i = 0; i < RS_WARPS; ++i) before += i < w ? wsum[i] : 0;
    lstart[tid] = before + x - cnt;
    run[tid] = before + x - cnt;
    __syncthreads();
    for (int r = 0; r < RS_ROUNDS; ++r) {
        for (int j = tid; j < RS_WARPS * 257; j += RS_THREADS) (&wcnt[0][0])[j] = 0;
        __syncthreads();
        const long i = tile + (long)r * RS_THREADS + tid;
        const bool valid = i < n;
        const uint32_t k = valid ? kin[i] : 0u;
        const uint32_t v = valid ? vin[i] : 0u;
        const int d = valid ? (int)((k >> shift) & 255u) : 256;
        const unsigned peers = __match_any_sync(FULL, d);
        const int rank = __popc(peers & lt);
        if (lane == __ffs(peers) - 1) wcnt[w][d] = __popc(peers);
        __syncthreads();
        {
            int s = run[tid];
#pragma unroll
            for (int ww = 0; ww < RS_WARPS; ++ww) {
                const int t = wcnt[ww][tid];
                wcnt[ww][tid] = s;
                s += t;
            }
            run[tid] = s;
        }
        __syncthreads();
        if (valid) {
            const int p = wcnt[w][d] + rank;
            sk[p] = k;
            sv[p] = v;
        }
        __syncthreads();
    }
    for (int j = tid; j < tile_n; j += RS_THREADS) {
        const uint32_t k = sk[j];
        const int d = (int)((k >> shift) & 255u);
        const int p = gbase[d] + (j - lstart[d]);
        kout[p] = k;
        vout[p] = sv[j];
    }
}

__global__ void k_count_keys(const uint32_t* keys, long n, int* counts) {
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        atomicAdd(&counts[keys[i]], 1);
}

// counts per key; slot[i] is the place the counter gave to i within its row, so that the scatter
// after the scan needs no atomics of its own
__global__ void k_count_slots(const uint32_t* keys, long n, int* counts, int* slot) {
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        slot[i] = atomicAdd(&counts[keys[i]], 1);
}

__global__ void k_scatter_slots(const uint32_t* keys, const int* slot, const int* rs, long n, uint32_t* out) {
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        if (slot[i] >= 0) out[rs[keys[i]] + slot[i]] = (uint32_t)i;
}

// one warp per row (grid-stride): the row's indices in ascending order (each placed by the number
// of smaller indices in the row: they are distinct), the row's key beside each (keys may be null),
// the longest row to *longest. Rows of more than SHORT_ROW_MAX indices are copied as they are.
__global__ void k_row_order(const int* rs, const uint32_t* idx, long K, uint32_t* order, uint32_t* keys, int* longest) {
    __shared__ int block_max;
    if (threadIdx.x == 0) block_max = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long nw = ((long)gridDim.x * blockDim.x) >> 5;
    int mx = 0;
    for (long r = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < K; r += nw) {
        const int b = rs[r], n = rs[r + 1] - b;
        mx = max(mx, n);
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            const uint32_t x = i < n ? idx[b + i] : 0u;
            int k = 0;
            if (n <= 32) {
                for (int j = 0; j < n; ++j) k += __shfl_sync(FULL, x, j) < x ? 1 : 0;
            } else if (n <= SHORT_ROW_MAX) {
                for (int j = 0; j < n; ++j) k += idx[b + j] < x ? 1 : 0;
            } else {
                k = i;
            }
            if (i < n) {
                order[b + k] = x;
                if (keys) keys[b + i] = (uint32_t)r;
            }
        }
    }
    if (lane == 0) atomicMax(&block_max, mx);
    __syncthreads();
    if (threadIdx.x == 0 && block_max > *(volatile int*)longest) atomicMax(longest, block_max);
}

__global__ void k_iota_u32(uint32_t* a, long n) {
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        a[i] = (uint32_t)i;
}

}  // namespace

int bits_for(uint32_t maxval) {
    int b = 1;
    while (b < 32 && (maxval >> b) != 0u) ++b;
    return b;
}

void exclusive_scan(const int* d_in, int* d_out, long n, int* d_total, cudaStream_t s) {
    if (n <= 0) {
        if (d_total) VSDMO_CUDA(cudaMemsetAsync(d_total, 0, sizeof(int), s));
        return;
    }
    scan(LoadInt{d_in}, StoreInt{d_out}, n, d_total, s);
}

template <int RS_ROUNDS>
static void radix_pass(const uint32_t* ka, const uint32_t* va, uint32_t* kb, uint32_t* vb, long n, int shift, int* counts, cudaStream_t s) {
    const int nTiles = (int)((n + RS_THREADS * RS_ROUNDS - 1) / (RS_THREADS * RS_ROUNDS));
    k_radix_hist<RS_ROUNDS><<<nTiles, RS_THREADS, 0, s>>>(ka, n, shift, counts, nTiles);
    VSDMO_CHECK_LAUNCH();
    exclusive_scan(counts, counts, 256L * nTiles, nullptr, s);
    k_radix_scatter<RS_ROUNDS><<<nTiles, RS_THREADS, 0, s>>>(ka, va, kb, vb, n, shift, counts, nTiles);
    VSDMO_CHECK_LAUNCH();
}

void radix_sort_pairs(uint32_t* keys, uint32_t* vals, long n, int bits, cudaStream_t s) {
    if (n <= 1 || bits <= 0) return;
    const bool small = n < RS_SMALL_N;
    const long tile = RS_THREADS * (small ? 4 : 16);
    DBuf<uint32_t> k2(n, s), v2(n, s);
    DBuf<int> counts(256L * ((n + tile - 1) / tile), s);
    uint32_t *ka = keys, *va = vals, *kb = k2.p, *vb = v2.p;
    for (int shift = 0; shift < bits; shift += 8) {
        (small ? radix_pass<4> : radix_pass<16>)(ka, va, kb, vb, n, shift, counts.p, s);
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    if (ka != keys) {
        VSDMO_CUDA(cudaMemcpyAsync(keys, ka, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
        VSDMO_CUDA(cudaMemcpyAsync(vals, va, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
    }
}

void compact_flags(const uint8_t* d_flags, long n, int* d_out_index, int* d_total, cudaStream_t s) {
    if (n <= 0) {
        if (d_total) VSDMO_CUDA(cudaMemsetAsync(d_total, 0, sizeof(int), s));
        return;
    }
    scan(LoadFlag{d_flags, 1}, StoreFlagged{d_out_index}, n, d_total, s);
}

void partition_flags(const uint8_t* d_flags, long n, int first_value, int* d_order, int* d_total, cudaStream_t s) {
    if (n <= 0) {
        VSDMO_CUDA(cudaMemsetAsync(d_total, 0, sizeof(int), s));
        return;
    }
    scan(LoadFlag{d_flags, first_value}, StorePartition{d_order}, n, d_total, s);
}

void rowptr_from_sorted(const uint32_t* d_sorted_keys, long n, int K, int* d_rowptr, cudaStream_t s) {
    DBuf<int> counts((long)K + 1, s);
    counts.zero();
    if (n > 0) {
        k_count_keys<<<grid_for(n, 256), 256, 0, s>>>(d_sorted_keys, n, counts.p);
        VSDMO_CHECK_LAUNCH();
    }
    exclusive_scan(counts.p, d_rowptr, (long)K + 1, nullptr, s);
}

void rows_from_slots(const uint32_t* d_keys, const int* d_slot, int* d_counts, long n, int K, int* d_rowptr,
                     uint32_t* d_rows, cudaStream_t s) {
    exclusive_scan(d_counts, d_rowptr, K, d_rowptr + K, s);
    if (n <= 0) return;
    k_scatter_slots<<<grid_for(n, 256), 256, 0, s>>>(d_keys, d_slot, d_rowptr, n, d_rows);
    VSDMO_CHECK_LAUNCH();
}

void order_short_rows(const int* d_rowptr, const uint32_t* d_rows, int K, uint32_t* d_order, uint32_t* d_keys,
                      int* d_longest, cudaStream_t s) {
    if (K <= 0) return;
    k_row_order<<<grid_for((long)K * 32, 256), 256, 0, s>>>(d_rowptr, d_rows, K, d_order, d_keys, d_longest);
    VSDMO_CHECK_LAUNCH();
}

void sort_short_rows(uint32_t* d_keys, uint32_t* d_order, long n, int K, int* d_rowptr, int* d_longest, cudaStream_t s) {
    if (K <= 0) return;
    DBuf<int> counts(K, s), slot(std::max(n, 1L), s);
    DBuf<uint32_t> rows(std::max(n, 1L), s);
    counts.zero();
    if (n > 0) {
        k_count_slots<<<grid_for(n, 256), 256, 0, s>>>(d_keys, n, counts.p, slot.p);
        VSDMO_CHECK_LAUNCH();
    }
    rows_from_slots(d_keys, slot.p, counts.p, n, K, d_rowptr, rows.p, s);
    order_short_rows(d_rowptr, rows.p, K, d_order, d_keys, d_longest, s);
}

void sort_long_rows(const uint32_t* d_keys, uint32_t* d_order, long n, int K, cudaStream_t s) {
    DBuf<uint32_t> k(n, s);
    VSDMO_CUDA(cudaMemcpyAsync(k.p, d_keys, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s));
    k_iota_u32<<<grid_for(n, 256), 256, 0, s>>>(d_order, n);
    VSDMO_CHECK_LAUNCH();
    radix_sort_pairs(k.p, d_order, n, bits_for((uint32_t)(K > 1 ? K - 1 : 1)), s);
}

cudaMemPool_t device_pool() {
    static std::mutex mu;
    static std::vector<cudaMemPool_t> pools;
    int dev = 0;
    VSDMO_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if ((int)pools.size() <= dev) pools.resize(dev + 1, nullptr);
    if (!pools[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        VSDMO_CUDA(cudaMemPoolCreate(&pool, &props));
        uint64_t keep = 8ull << 30;
        VSDMO_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        pools[dev] = pool;
    }
    return pools[dev];
}

}  // namespace vsdmo
