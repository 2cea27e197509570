// mesh_build.cu -- connectivity and colouring of tri / quad / tet / hex meshes on the GPU.
//
// Produces, bit for bit, the layout the reference's MeshTetGPU::init / MeshTriGPU::init build
// (mesh/MeshTetGPU.cu:35-42, mesh/MeshTriGPU.cu:37-50):
//   * boundary faces of a tet mesh: every tet face rotated smallest-index-first
//     (mesh/MeshGPUCommon.cu:1371-1410), sorted lexicographically, faces meeting their
//     opposite-oriented twin removed (k_markDuplicateTris, :56-74);
//   * vertex order [free surface by colour | feature surface by colour | inner by colour]
//     through stable partitions and stable colour sorts (mesh/MeshTetGPU.cu:241-295,
//     mesh/MeshTriGPU.cu:597-671), elements remapped after each step;
//   * halfedge CSR with boundary dummies, CCW fan order, opposite and next
//     (mesh/MeshTriGPU.cu:128-214, mesh/MeshGPUCommon.cu:96-135,211-285,565-620); quad meshes
//     the same with faces of four corners (mesh/MeshQuadGPU.cu), the fan walk stepping to the
//     corner two after the target (getThirdVertex, mesh/MeshGPUCommon.cu:149-162) and the
//     colouring adjacency holding both diagonals (:1067-1097);
//   * halfface CSR, rows in tetrahedron order (mesh/MeshTetGPU.cu:113-142); for hex meshes the
//     boundary quads (mesh/MeshHexGPU.cu:141-164), the all-pairs colouring graph of a hexahedron
//     and the halfhex CSR (mesh/MeshHexGPU.cu:116-139, mesh/MeshGPUCommon.cu:1334-1368);
//   * boundary / feature flags (dihedral > 20 deg, mesh/MeshGPUCommon.cu:466-495) and face /
//     vertex normals (:363-434).
// Elements keep the input's numbering until the end; one table of the elements around each vertex
// serves the boundary faces, the colouring and the halfface rows. Colouring follows the reference's JPL round
// rule (mesh/VertexColoring.cu:76-105): by default with seeded hash priorities, each vertex
// taking the smallest colour none of its higher-priority neighbours has (the greedy colouring in
// priority order, each vertex as soon as those neighbours are coloured); with VSDMO_COLOR_ROUNDS in the seed the colour is the
// round (the reference's rule) with the hashed priorities of the seed's other bits; with
// VSDMO_COLOR_REFERENCE the colour is the round and the priorities are the reference's own n - i
// (VertexColoring.cu:107-125).
#include "vsdmo_internal.cuh"
#include <climits>
#include <cmath>

namespace vsdmo {
namespace {

enum BuildErr { BE_OK = 0, BE_INDEX = 1, BE_NAN = 2, BE_DEGENERATE = 3, BE_NONMANIFOLD = 4,
                BE_FAN = 5, BE_FEATURE_START = 6 };

// n: the number of vertices coloured together (i is local to them)
__device__ __forceinline__ uint32_t priority(uint32_t i, uint32_t seed, uint32_t n) {
    if (seed == VSDMO_COLOR_REFERENCE) return n - i;
    seed &= ~VSDMO_COLOR_ROUNDS;
    uint32_t h = i + seed * 0x9E3779B9u;
    h ^= h >> 16; h *= 0x85EBCA6Bu;
    h ^= h >> 13; h *= 0xC2B2AE35u;
    h ^= h >> 16;
    return h;
}

// the halfedge fans are walked by one thread per vertex in time quadratic in the fan's length
// (k_ccw, like the reference's k_sortCCWDummyOpposite): longer fans are refused
[[noreturn]] void throw_long_fan() {
    throw Error(VSDMO_E_VALENCE, "a vertex has more than " + std::to_string(SHORT_ROW_MAX) + " halfedges");
}

#define GRID_STRIDE(i, n) for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (long)gridDim.x * blockDim.x)
constexpr unsigned FULL = 0xffffffffu;

// copies the input, checks it and counts each vertex's elements; slot: the place of an element corner
// among its vertex's (-1: index out of range). The counter's old value is that place, so one pass of
// atomics serves the whole vertex-to-element table.
__global__ void k_input(const float* xyz, int nV, const int* elems, long nIdx, float4* pos, int* orig, int* cur,
                        int* out, int* counts, int* slot, int* err, int* nonzero_z) {
    GRID_STRIDE(i, nV) {
        float x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
        if (!isfinite(x) || !isfinite(y) || !isfinite(z)) atomicMax(err, BE_NAN);
        if (z != 0.f) *nonzero_z = 1;
        pos[i] = make_float4(x, y, z, 0.f);
        orig[i] = cur[i] = (int)i;
    }
    GRID_STRIDE(i, nIdx) {
        int v = elems[i];
        out[i] = v;
        const bool bad = v < 0 || v >= nV;
        if (bad) atomicMax(err, BE_INDEX);
        slot[i] = bad ? -1 : atomicAdd(&counts[v], 1);
    }
}

__global__ void k_iota(uint32_t* a, long n) { GRID_STRIDE(i, n) a[i] = (uint32_t)i; }

template <class T>
__global__ void k_gather(const T* src, const uint32_t* idx, T* dst, long n) { GRID_STRIDE(i, n) dst[i] = src[idx[i]]; }

__global__ void k_gather_key(const uint32_t* src, const uint32_t* idx, uint32_t* dst, long n) {
    GRID_STRIDE(i, n) dst[i] = src[idx[i]];
}

// ---- tetrahedral boundary ---------------------------------------------------------------
__device__ __forceinline__ void smallest_first(int a, int b, int c, uint32_t* o) {
    if (a < b && a < c) { o[0] = a; o[1] = b; o[2] = c; }
    else if (b < a && b < c) { o[0] = b; o[1] = c; o[2] = a; }
    else { o[0] = c; o[1] = a; o[2] = b; }
}

// One warp per vertex a (grid-stride): the faces whose first vertex is a, from the tets around a
// (rs, inc: element corners 4 t + j by vertex). Corner j of tet t owns the faces of t that
// smallest_first starts at j, so every face is looked at once. Face (a, b, c) is a boundary face
// unless the row also holds its twin (a, c, b) (k_markDuplicateTris, mesh/MeshGPUCommon.cu:56-74); an
// exact repeat is a non-manifold input. A boundary face takes its place among the row's boundary faces in
// (b, c) order, so rows in vertex order give the lexicographic order of a sort; rec collects
// them in any order as (b << 32 | c, a << 32 | place) and u counts them per row.
// Bound by the instructions per face: rows of up to 32 faces (22 on average) pair them with one match
// over the warp, longer ones scan the row; rows live in shared memory (up to FACE_CAP faces; longer ones in
// their own part of spill). Five passes over lists of all faces in global memory before: 180 us for
// 663,552 tets with cold caches, 58 us now (87 us with the scan for every row).
constexpr int FACE_CAP = 160;
constexpr int FACE_WARPS = 4;
__global__ void __launch_bounds__(FACE_WARPS * 32)
k_tet_boundary(const int* __restrict__ rs, const uint32_t* __restrict__ inc, const int4* __restrict__ tets, long K,
               const int* input_err, unsigned long long* spill, uint8_t* spill_flag, int* spill_used, int* u,
               ulonglong2* rec, int* nrec, uint8_t* isB2, int* err, int* longest) {
    __shared__ unsigned long long sf[FACE_WARPS][FACE_CAP];
    __shared__ uint8_t sb[FACE_WARPS][FACE_CAP];
    if (*input_err != BE_OK) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const long nw = (long)gridDim.x * FACE_WARPS;
    for (long r = (long)blockIdx.x * FACE_WARPS + warp; r < K; r += nw) {
        const int b0 = rs[r], m = rs[r + 1] - b0;
        unsigned long long* f = sf[warp];
        uint8_t* bnd = sb[warp];
        int n = 0;
        for (int pass = 0; pass < 2; ++pass) {
            n = 0;
            for (int i0 = 0; i0 < m; i0 += 32) {
                // lane: one tet and the three faces of corner j (all but the one opposite)
                const bool has = i0 + lane < m;
                const uint32_t e = has ? inc[b0 + i0 + lane] : 0u;
                const int j = e & 3, skip = j == 0 ? 2 : (j == 1 ? 3 : (j == 2 ? 1 : 0));
                const int4 t = tets[e >> 2];
#pragma unroll
                for (int face = 0; face < 4; ++face) {
                    const int a = face == 0 ? t.z : (face == 2 ? t.y : t.x), b = face == 2 ? t.z : (face == 3 ? t.w : t.y),
                              c = face == 0 ? t.x : (face == 3 ? t.z : t.w);
                    const int first = a < b && a < c ? 0 : (b < a && b < c ? 1 : 2);
                    // the place in the tet of the face's first vertex
                    const int at0 = face == 0 ? 2 - first : face == 1 ? (first == 2 ? 3 : first) : face == 2 ? 1 + first
                                  : (first == 0 ? 0 : 4 - first);
                    const bool own = has && face != skip && at0 == j;
                    const unsigned mask = __ballot_sync(FULL, own);
                    const int at = n + __popc(mask & lt);
                    if (own && (pass == 1 || at < FACE_CAP)) {
                        uint32_t o[3];
                        smallest_first(a, b, c, o);
                        f[at] = ((unsigned long long)o[1] << 32) | o[2];
                    }
                    n += __popc(mask);
                }
            }
            if (pass == 1 || n <= FACE_CAP || n > SHORT_ROW_MAX) break;
            int at = 0;
            if (lane == 0) at = atomicAdd(spill_used, n);
            at = __shfl_sync(FULL, at, 0);
            f = spill + at;
            bnd = spill_flag + at;
        }
        if (n > SHORT_ROW_MAX) {
            if (lane == 0) atomicMax(longest, n);
            continue;
        }
        __syncwarp();
        int cnt = 0;
        if (n <= 32) {
            // one face per lane: its peers hold the same two vertices, in this order (a repeat) or the other (its twin)
            const unsigned long long x = lane < n ? f[lane] : 0ull;
            const unsigned p = (unsigned)(x >> 32), q = (unsigned)x;
            const unsigned up = __ballot_sync(FULL, p < q), self = 1u << lane;
            const unsigned peers = __match_any_sync(FULL, lane < n ? ((unsigned long long)min(p, q) << 32) | max(p, q)
                                                                   : ~(unsigned long long)lane);
            const unsigned same = (p < q ? up : ~up) & peers;
            if (lane < n) {
                if (same & ~self) atomicMax(err, BE_NONMANIFOLD);
                bnd[lane] = peers == same ? 1 : 0;
                cnt = bnd[lane];
            }
        } else {
            for (int i = lane; i < n; i += 32) {
                const unsigned long long x = f[i], twin = (x << 32) | (x >> 32);
                bool paired = false, repeat = false;
                for (int j = 0; j < n; ++j) {
                    const unsigned long long y = f[j];
                    repeat |= y == x && j != i;
                    paired |= y == twin && j != i;
                }
                if (repeat) atomicMax(err, BE_NONMANIFOLD);
                bnd[i] = paired ? 0 : 1;
                cnt += paired ? 0 : 1;
            }
        }
        cnt = __reduce_add_sync(FULL, cnt);
        if (lane == 0) u[r] = cnt;
        if (cnt) {
            __syncwarp();
            int at = 0;
            if (lane == 0) at = atomicAdd(nrec, cnt);
            at = __shfl_sync(FULL, at, 0);
            for (int i = lane; i < n; i += 32) {
                if (!bnd[i]) continue;
                const unsigned long long x = f[i];
                int k = 0;
                for (int j = 0; j < n; ++j) k += (bnd[j] && f[j] < x) ? 1 : 0;
                // a repeat leaves two faces on one place: the build ends in an error, the list stays in bounds
                rec[at + k] = make_ulonglong2(x, ((unsigned long long)r << 32) | (unsigned)k);
                isB2[r] = 1; isB2[x >> 32] = 1; isB2[x & 0xffffffffull] = 1;
            }
        }
        __syncwarp();
    }
}

__global__ void k_face_emit(const ulonglong2* rec, int nB, const int* offs, int* tris) {
    GRID_STRIDE(i, nB) {
        const ulonglong2 x = rec[i];
        const int a = (int)(x.y >> 32);
        const long p = (long)offs[a] + (int)(x.y & 0xffffffffull);
        tris[3 * p] = a; tris[3 * p + 1] = (int)(x.x >> 32); tris[3 * p + 2] = (int)(x.x & 0xffffffffull);
    }
}

// ---- hexahedral boundary (MeshHexGPU::initBoundary2D, mesh/MeshHexGPU.cu:141-164) --------------
// getQuadSmallestFirst: rotate so that the smallest index comes first (mesh/MeshGPUCommon.cu:37-54)
__device__ __forceinline__ void quad_smallest_first(int a, int b, int c, int d, uint32_t* o) {
    if (b < a && b < c && b < d) { o[0] = b; o[1] = c; o[2] = d; o[3] = a; }
    else if (c < a && c < b && c < d) { o[0] = c; o[1] = d; o[2] = a; o[3] = b; }
    else if (d < a && d < b && d < c) { o[0] = d; o[1] = a; o[2] = b; o[3] = c; }
    else { o[0] = a; o[1] = b; o[2] = c; o[3] = d; }
}

// the six faces of a hexahedron (k_constructQuadsFromHexahedra, mesh/MeshGPUCommon.cu:1412-1430)
__global__ void k_hex_faces(const int* hexes, int nH, uint32_t* f0, uint32_t* f1, uint32_t* f2, uint32_t* f3) {
    const int F[6][4] = { {0, 1, 2, 3}, {1, 5, 6, 2}, {3, 2, 6, 7}, {4, 0, 3, 7}, {1, 0, 4, 5}, {5, 4, 7, 6} };
    GRID_STRIDE(t, nH) {
        const int* v = hexes + 8 * t;
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            uint32_t o[4];
            quad_smallest_first(v[F[f][0]], v[F[f][1]], v[F[f][2]], v[F[f][3]], o);
            f0[6 * t + f] = o[0]; f1[6 * t + f] = o[1]; f2[6 * t + f] = o[2]; f3[6 * t + f] = o[3];
        }
    }
}

__device__ __forceinline__ int cmp4(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1,
                                    uint32_t b2, uint32_t b3) {
    if (a0 != b0) return a0 < b0 ? -1 : 1;
    if (a1 != b1) return a1 < b1 ? -1 : 1;
    if (a2 != b2) return a2 < b2 ? -1 : 1;
    if (a3 != b3) return a3 < b3 ? -1 : 1;
    return 0;
}

// quads sorted lexicographically: (a,b,c,d) with b<d pairs with (a,d,c,b) (k_markDuplicateQuads)
__global__ void k_pair_quads(const uint32_t* s0, const uint32_t* s1, const uint32_t* s2, const uint32_t* s3, long nF,
                             uint8_t* paired, int* err) {
    GRID_STRIDE(i, nF) {
        const uint32_t a = s0[i], b = s1[i], c = s2[i], d = s3[i];
        if (i + 1 < nF && s0[i + 1] == a && s1[i + 1] == b && s2[i + 1] == c && s3[i + 1] == d) atomicMax(err, BE_NONMANIFOLD);
        if (b < d) {
            long lo = i + 1, hi = nF;
            while (lo < hi) {
                const long mid = (lo + hi) >> 1;
                if (cmp4(s0[mid], s1[mid], s2[mid], s3[mid], a, d, c, b) < 0) lo = mid + 1; else hi = mid;
            }
            if (lo < nF && s0[lo] == a && s1[lo] == d && s2[lo] == c && s3[lo] == b) { paired[i] = 1; paired[lo] = 1; }
        }
    }
}

__global__ void k_emit_boundary_quads(const int* idx, int nB, const uint32_t* s0, const uint32_t* s1, const uint32_t* s2,
                                      const uint32_t* s3, int* quads, uint8_t* isB2) {
    GRID_STRIDE(i, nB) {
        const int j = idx[i];
        const int a = s0[j], b = s1[j], c = s2[j], d = s3[j];
        quads[4 * i] = a; quads[4 * i + 1] = b; quads[4 * i + 2] = c; quads[4 * i + 3] = d;
        isB2[a] = 1; isB2[b] = 1; isB2[c] = 1; isB2[d] = 1;
    }
}

// halfhex of corner j: the other seven corners (k_constructHalfhexesNew, mesh/MeshGPUCommon.cu:1334-1368),
// two int4 per halfhex (the eighth value is -1)
// the rows of inc (element corners by original vertex) in the final vertex order: row i is that of vertex orig[i]
__global__ void k_halfhexes(const int* rs, const uint32_t* inc, const int* orig, const int* rowptr, int nV,
                            const int* hexes, int4* hh) {
    const int H[8][7] = { {1, 2, 3, 4, 5, 6, 7}, {5, 6, 2, 0, 4, 7, 3}, {6, 7, 3, 1, 5, 4, 0}, {7, 4, 0, 2, 6, 5, 1},
                          {0, 3, 7, 5, 1, 2, 6}, {4, 7, 6, 1, 0, 3, 2}, {5, 4, 7, 2, 1, 0, 3}, {6, 5, 4, 3, 2, 1, 0} };
    const int lane = threadIdx.x & 7;
    const long nw = ((long)gridDim.x * blockDim.x) >> 3;
    for (long r = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 3; r < nV; r += nw) {
        const int src = rs[orig[r]], dst = rowptr[r], n = rowptr[r + 1] - dst;
        for (int q = lane; q < n; q += 8) {
            const int e = (int)inc[src + q], t = e >> 3, j = e & 7;
            const int* v = hexes + 8L * t;
            const long i = dst + q;
            hh[2 * i] = make_int4(v[H[j][0]], v[H[j][1]], v[H[j][2]], v[H[j][3]]);
            hh[2 * i + 1] = make_int4(v[H[j][4]], v[H[j][5]], v[H[j][6]], -1);
        }
    }
}

__global__ void k_not(const uint8_t* f, uint8_t* o, long n) { GRID_STRIDE(i, n) o[i] = f[i] ? 0 : 1; }

// ---- permutations -----------------------------------------------------------------------
// New vertex order: position start + i comes from start + order[i] for i < num, the others stay. One pass moves the
// positions, the original indices with their inverse and up to two flag arrays (of nf0 / nf1
// vertices) and leaves the map for the remap of index arrays.
__global__ void k_permute(const int* order, int start, int num, int nTot, const float4* pin, float4* pout,
                          const int* oin, int* oout, int* cur_of_orig, int* new_of_old, const uint8_t* f0, uint8_t* g0, int nf0,
                          const uint8_t* f1, uint8_t* g1, int nf1) {
    GRID_STRIDE(i, nTot) {
        const int o = i >= start && i < start + num ? start + order[i - start] : (int)i;
        pout[i] = pin[o];
        const int og = oin[o];
        oout[i] = og;
        cur_of_orig[og] = (int)i;
        new_of_old[o] = (int)i;
        if (i < nf0) g0[i] = f0[o];
        if (i < nf1) g1[i] = f1[o];
    }
}

__global__ void k_remap(int* idx, long n, const int* new_of_old) {
    GRID_STRIDE(i, n) idx[i] = new_of_old[idx[i]];
}

// ---- JPL colouring ---------------------------------------------------------------------------
// The vertices of [lo, lo + num) that share an element are neighbours, and every vertex waits for its
// neighbours of higher priority only: its colour is the smallest one none of them has (first fit), or
// 1 + the largest of them (round colours: the JPL round it would be coloured in). Both are
// functions of those neighbours' colours alone, so a vertex may be coloured as soon as they are,
// in any order and without rounds, and the colours are those of the round-by-round rule.
//
// k_wait_lists: one warp per vertex, its higher-priority neighbours (places in the range) from the
// elements around it to list[(k - 1) * rs[original vertex]], their number beside the row start in
// info. Neighbours seen more than once are dropped by a small table that keeps the last value of
// each hash; the few it lets through twice change nothing. Bound by the latency of its gathers
// (47 us with cold caches for the 103,823 inner vertices of 663,552 tets); writing, bucketing, deduplicating
// and copying all neighbour pairs as a CSR before: 445 us.
constexpr int WAIT_TABLE = 128;
template <int KC>
__global__ void __launch_bounds__(128)
k_wait_lists(const int* __restrict__ rs, const uint32_t* __restrict__ inc, const int* __restrict__ elems,
             const int* __restrict__ orig_of_cur, const int* __restrict__ cur_of_orig, int lo, int num, uint32_t seed,
             int* list, int2* info, int* colors) {
    __shared__ int table[4][WAIT_TABLE];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const long nw = (long)gridDim.x * 4;
    for (long v = (long)blockIdx.x * 4 + warp; v < num; v += nw) {
        for (int j = lane; j < WAIT_TABLE; j += 32) table[warp][j] = -1;
        const int o = orig_of_cur[lo + v], b0 = rs[o], m = (KC - 1) * (rs[o + 1] - b0);
        int* out = list + (long)(KC - 1) * b0;
        const uint32_t pv = priority((uint32_t)v, seed, (uint32_t)num);
        int n = 0;
        __syncwarp();
        for (int i0 = 0; i0 < m; i0 += 32) {
            const int i = i0 + lane;
            bool take = false;
            int w = 0;
            if (i < m) {
                const uint32_t e = inc[b0 + i / (KC - 1)];
                const uint32_t j = e % KC, c = (j + 1 + i % (KC - 1)) % KC;
                w = cur_of_orig[elems[e - j + c]] - lo;
                if (w >= 0 && w < num && w != (int)v && priority((uint32_t)w, seed, (uint32_t)num) >= pv)
                    take = atomicExch(&table[warp][(w * 0x9E3779B1u) >> 25], w) != w;
            }
            const unsigned mask = __ballot_sync(FULL, take);
            if (take) out[n + __popc(mask & lt)] = w;
            n += __popc(mask);
        }
        if (lane == 0) {
            info[v] = make_int2(b0, n);
            colors[v] = -1;
        }
        __syncwarp();
    }
}

// One thread per vertex: looks COLOUR_TRIES times whether the vertices it waits for have their
// colours (going on from the first one that had none) and then takes its own. What is left after
// the tries is counted in *remaining and taken up by the next launch; prev: the count of the launch
// before (null for the first); when it is 0 nothing is left. A launch always colours the uncoloured vertex
// of highest priority, so the launches end whatever the order the blocks run in. hist counts
// the colours below 256, maxc collects the largest. Chains of waiting vertices pass within one
// launch at the latency of a read through L2 (45 + 24 + 12 us for 103,823 vertices); a launch per
// round before: 32 launches of up to 14 us.
constexpr int COLOUR_TRIES = 32;
__global__ void __launch_bounds__(256)
k_colour(int num, const int* __restrict__ list, int per_slot, const int2* __restrict__ info, int first_fit, int* colors, int* remaining,
         const int* prev, int* maxc, int* hist) {
    if (prev && *prev == 0) return;
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    volatile int* col = colors;
    bool todo = v < num && col[v] < 0;
    int colour = -1;
    if (__any_sync(FULL, todo)) {
        const int* p = nullptr;
        int n = 0, at = 0, mx = -1;
        unsigned long long used = 0ull;
        if (todo) {
            const int2 w = info[v];
            p = list + (long)per_slot * w.x;
            n = w.y;
        }
        for (int t = 0; t < COLOUR_TRIES && __any_sync(FULL, todo && colour < 0); ++t) {
            if (!todo || colour >= 0) continue;
            while (at < n) {
                int c[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) c[j] = at + j < n ? col[p[at + j]] : -2;
                int j = 0;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (j != q || c[q] < 0) continue;
                    if (c[q] < 64) used |= 1ull << c[q];
                    mx = max(mx, c[q]);
                    ++j;
                }
                at += j;
                if (j < 4) break;
            }
            if (at < n) continue;
            if (!first_fit) {
                colour = mx + 1;
            } else if (~used) {
                colour = __ffsll((long long)~used) - 1;
            } else {
                for (colour = 64;; ++colour) {
                    bool taken = false;
                    for (int e = 0; e < n && !taken; ++e) taken = col[p[e]] == colour;
                    if (!taken) break;
                }
            }
            col[v] = colour;
        }
        __syncwarp();
    }
    const unsigned left = __ballot_sync(FULL, todo && colour < 0);
    const int lane = threadIdx.x & 31;
    if (left && lane == 0) atomicAdd(remaining, __popc(left));
    const unsigned same = __match_any_sync(FULL, colour);
    if (colour >= 0 && lane == __ffs(same) - 1) {
        if (colour < 256) atomicAdd(&hist[colour], __popc(same));
        if (colour > *(volatile int*)maxc) atomicMax(maxc, colour);
    }
}

// offs[c] = lo + the vertices of the colours below c (nc <= 256 colours; one block of 256 threads)
__global__ void k_colour_offsets(const int* hist, int nc, int lo, int* offs) {
    __shared__ int h[256];
    const int t = threadIdx.x;
    h[t] = t < nc ? hist[t] : 0;
    __syncthreads();
    int s = lo;
    for (int i = 0; i < t; ++i) s += h[i];
    if (t < nc) offs[t] = s;
    if (t == nc - 1) offs[nc] = s + h[t];
}

__global__ void k_add_const(int* a, long n, int v) { GRID_STRIDE(i, n) a[i] += v; }

// ---- surface ------------------------------------------------------------------------------------
// face normal from corners 0, 1 and 2 (triangles) or 0, 1 and 3 (quads)
__global__ void k_face_normals(const int* tris, int fk, int nTris, const float4* pos, float* fn, int* err) {
    GRID_STRIDE(t, nTris) {
        const int* f = tris + (long)fk * t;
        float4 p0 = pos[f[0]], p1 = pos[f[1]], p2 = pos[f[fk == 4 ? 3 : 2]];
        float e0x = p1.x - p0.x, e0y = p1.y - p0.y, e0z = p1.z - p0.z;
        float e1x = p2.x - p0.x, e1y = p2.y - p0.y, e1z = p2.z - p0.z;
        if (err) {
            float l0 = sqrtf(e0x * e0x + e0y * e0y + e0z * e0z);
            float l1 = sqrtf(e1x * e1x + e1y * e1y + e1z * e1z);
            if (l0 < 1e-6f || l1 < 1e-6f) atomicMax(err, BE_DEGENERATE);
        }
        float nx = e0y * e1z - e0z * e1y, ny = e0z * e1x - e0x * e1z, nz = e0x * e1y - e0y * e1x;
        float len = sqrtf(nx * nx + ny * ny + nz * nz);
        fn[3 * t] = nx / len; fn[3 * t + 1] = ny / len; fn[3 * t + 2] = nz / len;
    }
}

// first-pass halfedges from the sorted (src, fk*t+j) pairs
__global__ void k_he_records(const uint32_t* order, long nHE, const int* tris, int fk, int4* he) {
    GRID_STRIDE(i, nHE) {
        int e = (int)order[i], t = e / fk, j = e % fk;
        he[i] = make_int4(tris[(long)fk * t + (j + 1) % fk], -1, t, 0);
    }
}

// opposite = last halfedge of the target's row that points back to the source
// (longest: the rows' maximum; above SHORT_ROW_MAX the build ends in an error and nothing is searched)
__global__ void k_opposite(const uint32_t* srcs, int4* he, long nHE, const int* rowptr, const int* longest) {
    if (*longest > SHORT_ROW_MAX) return;
    GRID_STRIDE(i, nHE) {
        int src = (int)srcs[i], dst = he[i].x, opp = -1;
        for (int q = rowptr[dst]; q < rowptr[dst + 1]; ++q) if (he[q].x == src) opp = q;
        he[i].y = opp;
    }
}

__global__ void k_flags_b1_feat(const uint32_t* srcs, const int4* he, long nHE, const float* fn, uint8_t* isB1,
                                uint8_t* isFeat, int flat, int* nOpen, const int* longest) {
    if (*longest > SHORT_ROW_MAX) return;
    GRID_STRIDE(i, nHE) {
        int src = (int)srcs[i];
        int4 h = he[i];
        if (h.y == -1) {
            atomicAdd(nOpen, 1);
            isB1[src] = 1;
            if (!flat) { isFeat[src] = 1; isFeat[h.x] = 1; }
            continue;
        }
        if (flat) continue;
        const float* f1 = fn + 3 * (long)h.z;
        const float* f2 = fn + 3 * (long)he[h.y].z;
        float dot = f1[0] * f2[0] + f1[1] * f2[1] + f1[2] * f2[2];
        float len = sqrtf((f1[0] * f1[0] + f1[1] * f1[1] + f1[2] * f1[2]) * (f2[0] * f2[0] + f2[1] * f2[1] + f2[2] * f2[2]));
        // the reference keeps the angle as a float (float angle = 180.f / M_PI * acosf(..),
        // MeshGPUCommon.cu:485-488): the double product is rounded before the compare
        const float angle = (float)(180.0 / 3.14159265358979323846 * (double)acosf(dot / len));
        if (angle > 20.f) { isFeat[src] = 1; isFeat[h.x] = 1; }
    }
}

__global__ void k_copy_u8(const uint8_t* a, uint8_t* b, long n) { GRID_STRIDE(i, n) b[i] = a[i]; }

__global__ void k_dummy_flags(const int4* he, long n, uint8_t* f) { GRID_STRIDE(i, n) f[i] = he[i].y == -1 ? 1 : 0; }

// real halfedges (sorted) followed by the dummies in the sorted order of their twins
__global__ void k_with_dummies(const uint32_t* srcs, const int4* he, long nHE1, const int* didx, int nD,
                               uint32_t* keys, int4* rec) {
    GRID_STRIDE(i, nHE1) { keys[i] = srcs[i]; rec[i] = make_int4(he[i].x, -1, he[i].z, 0); }
    GRID_STRIDE(j, nD) {
        int i = didx[j];
        keys[nHE1 + j] = (uint32_t)he[i].x;
        rec[nHE1 + j] = make_int4((int)srcs[i], -1, -1, 0);
    }
}

__device__ __forceinline__ int third_vertex(const int* t, int src, int dst) {
    if (t[0] != src && t[0] != dst) return t[0];
    if (t[1] != src && t[1] != dst) return t[1];
    return t[2];
}

// the corner two after dst (getThirdVertex for quads)
__device__ __forceinline__ int third_vertex_quad(const int* q, int dst) {
    if (dst == q[1]) return q[3];
    if (dst == q[2]) return q[0];
    if (dst == q[3]) return q[1];
    return q[2];
}

__global__ void k_ccw(int nS, const int* rowptr, const int4* in, int4* out, const uint8_t* isB1, const uint8_t* isFeat,
                      const int* tris, int fk, int* err, const int* longest) {
    if (*longest > SHORT_ROW_MAX) return;
    GRID_STRIDE(src, nS) {
        const int start = rowptr[src], n = rowptr[src + 1] - start;
        if (n == 0) { atomicMax(err, BE_FAN); continue; }
        int outPos = 0;
        int4 h = in[start];
        bool bad = false;
        if (isB1[src]) {
            int j = 0;
            while (true) {
                if (h.y < 0) { bad = true; break; }
                if (in[h.y].z == -1) break;
                if (++j == n) { bad = true; break; }
                h = in[start + j];
            }
        } else if (isFeat[src]) {
            h.x = INT_MAX;
            for (int j = 0; j < n; ++j) {
                int4 t = in[start + j];
                if (isFeat[t.x] && t.x < h.x) h = t;
            }
            if (h.x == INT_MAX) { atomicMax(err, BE_FEATURE_START); continue; }
        } else {
            for (int i = 1; i < n; ++i) { int4 t = in[start + i]; if (t.x < h.x) h = t; }
        }
        if (bad) { atomicMax(err, BE_FAN); continue; }
        out[start + outPos++] = h;
        bool found;
        do {
            int currDst = h.x, currTri = h.z;
            if (currTri == -1) { bad = true; break; }
            int nextVert = fk == 4 ? third_vertex_quad(tris + 4 * (long)currTri, currDst)
                                   : third_vertex(tris + 3 * (long)currTri, (int)src, currDst);
            found = false;
            for (int j = 0; j < n; ++j) {
                int4 t = in[start + j];
                if (t.x == nextVert) {
                    if (outPos >= n) { bad = true; break; }
                    found = true; h = t; out[start + outPos++] = h;
                }
            }
            if (bad) break;
        } while (found && outPos < n);
        if (bad || outPos != n) atomicMax(err, BE_FAN);
    }
}

__global__ void k_opp_next(int nS, const int* rowptr, int4* he, const int* err, const int* longest) {
    if (*err != BE_OK || *longest > SHORT_ROW_MAX) return;
    GRID_STRIDE(v, nS) {
        for (int i = rowptr[v]; i < rowptr[v + 1]; ++i) {
            int4 h = he[i];
            int opp = -1, nxt = h.w;
            for (int q = rowptr[h.x]; q < rowptr[h.x + 1]; ++q) {
                int4 o = he[q];
                if (o.x == (int)v) opp = q;
                if (o.z == h.z) nxt = q;
            }
            he[i].y = opp; he[i].w = nxt;
        }
    }
}

__global__ void k_vertex_normals(int nS, const int* rowptr, const int4* he, const float* fn, float* vn) {
    GRID_STRIDE(v, nS) {
        float nx = 0.f, ny = 0.f, nz = 0.f;
        for (int i = rowptr[v]; i < rowptr[v + 1]; ++i) {
            int f = he[i].z;
            if (f != -1) { nx += fn[3 * f]; ny += fn[3 * f + 1]; nz += fn[3 * f + 2]; }
        }
        float len = sqrtf(nx * nx + ny * ny + nz * nz);
        vn[3 * v] = nx / len; vn[3 * v + 1] = ny / len; vn[3 * v + 2] = nz / len;
    }
}

// ---- halffaces ------------------------------------------------------------------------------------
// the rows of inc (element corners by original vertex) in the final vertex order: row i is that of vertex orig[i]
__global__ void k_halffaces(const int* rs, const uint32_t* inc, const int* orig, const int* rowptr, int nV,
                            const int4* tets, int4* hf) {
    const int lane = threadIdx.x & 7;
    const long nw = ((long)gridDim.x * blockDim.x) >> 3;
    for (long r = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 3; r < nV; r += nw) {
        const int src = rs[orig[r]], dst = rowptr[r], n = rowptr[r + 1] - dst;
        for (int q = lane; q < n; q += 8) {
            const uint32_t e = inc[src + q];
            const int t = e >> 2, j = e & 3;
            const int4 v = tets[t];
            int4 o;
            if (j == 0) o = make_int4(v.y, v.z, v.w, t);
            else if (j == 1) o = make_int4(v.x, v.w, v.z, t);
            else if (j == 2) o = make_int4(v.x, v.y, v.w, t);
            else o = make_int4(v.x, v.z, v.y, t);
            hf[dst + q] = o;
        }
    }
}

// row lengths in the final vertex order
__global__ void k_row_lengths(const int* rs, const int* orig, int nV, int* len) {
    GRID_STRIDE(i, nV) len[i] = rs[orig[i] + 1] - rs[orig[i]];
}

inline int G(long n) { return grid_for(n, 256); }

void check_err(int e, const char* stage) {
    switch (e) {
    case BE_OK: return;
    case BE_INDEX: throw Error(VSDMO_E_ARG, std::string(stage) + ": element index out of range");
    case BE_NAN: throw Error(VSDMO_E_NAN, std::string(stage) + ": non-finite vertex coordinate");
    case BE_DEGENERATE: throw Error(VSDMO_E_ARG, std::string(stage) + ": degenerate triangle (edge shorter than 1e-6)");
    case BE_NONMANIFOLD: throw Error(VSDMO_E_NONMANIFOLD, std::string(stage) + ": a face occurs twice with the same orientation");
    case BE_FAN: throw Error(VSDMO_E_NONMANIFOLD, std::string(stage) + ": a vertex fan is open or non-manifold");
    case BE_FEATURE_START: throw Error(VSDMO_E_NONMANIFOLD, std::string(stage) + ": feature vertex without feature neighbour");
    default: throw Error(VSDMO_E_CUDA, std::string(stage) + ": unknown build error");
    }
}

// what the build's kernels report, read by the host a few times in one piece
struct BuildStatus {
    int input_err;       // BE_* of the input
    int nonzero_z;
    int longest_elems;   // elements around one vertex
    int face_err, face_rows, spill, nB, nS;   // boundary faces: error, longest refused row, ..., faces, boundary vertices
    int surf_err, longest_he, nOpen, nFree;   // faces: error; halfedges of one vertex; boundary halfedges; free vertices
    int fan_err, longest_full;                // fans: error, halfedges of one vertex with the dummies
};
struct ColourStatus {
    int remaining[4];
    int maxc;
    int hist[256];
};

// Shared state of one build.
struct Builder {
    Mesh& m;
    cudaStream_t s;
    DBuf<int> orig_of_cur, cur_of_orig;
    DBuf<int> inc_rs;                 // elements around each vertex (original numbering): rows and
    DBuf<uint32_t> inc;               // element corners k e + j
    DBuf<BuildStatus> st;
    explicit Builder(Mesh& mm) : m(mm), s(mm.stream) {}

    BuildStatus status() { return read_scalar(st.p, s); }
    int* at(int BuildStatus::* f) { return &(st.p->*f); }

    // apply a permutation of range [start, start+num) given as order_local (new -> old, local) to the vertices and the
    // surface; the elements keep the original numbering until finish_elems()
    void permute_range(const int* order_local, int start, int num, std::vector<DBuf<uint8_t>*> flags) {
        const int nTot = m.nV;
        DBuf<int> noo(nTot, s), o2(nTot, s);
        DBuf<float4> p2(nTot, s);
        DBuf<uint8_t> g[2];
        const uint8_t* f[2] = { nullptr, nullptr };
        for (size_t i = 0; i < flags.size(); ++i) {
            if (!flags[i]->p) continue;
            f[i] = flags[i]->p;
            g[i].alloc(flags[i]->n, s);
        }
        k_permute<<<G(nTot), 256, 0, s>>>(order_local, start, num, nTot, m.pos.p, p2.p, orig_of_cur.p, o2.p, cur_of_orig.p, noo.p,
                                          f[0], g[0].p, (int)g[0].n, f[1], g[1].p, (int)g[1].n);
        VSDMO_CHECK_LAUNCH();
        m.pos = std::move(p2);
        orig_of_cur = std::move(o2);
        for (size_t i = 0; i < flags.size(); ++i)
            if (f[i]) *flags[i] = std::move(g[i]);
        const long nt = m.tris.p ? (long)m.fk * m.nTris : 0;
        if (nt > 0) {
            k_remap<<<G(nt), 256, 0, s>>>(m.tris.p, nt, noo.p);
            VSDMO_CHECK_LAUNCH();
        }
    }

    // colour the range [lo, lo+num), sort it by colour; returns the number of colours
    int color_range(int lo, int num, std::vector<int>& offs_host, DBuf<int>& offs_dev, std::vector<DBuf<uint8_t>*> flags) {
        const int first_fit = m.seed != VSDMO_COLOR_REFERENCE && !(m.seed & VSDMO_COLOR_ROUNDS) ? 1 : 0;
        DBuf<int> colors(num, s), list(std::max<size_t>((size_t)(m.k - 1) * inc.n, 1), s);
        DBuf<int2> info(num, s);
        DBuf<ColourStatus> cs(1, s);
        cs.zero();
        auto lists = m.k == 3 ? k_wait_lists<3> : m.k == 4 ? k_wait_lists<4> : k_wait_lists<8>;
        lists<<<grid_for(32L * num, 128), 128, 0, s>>>(inc_rs.p, inc.p, m.elems.p, orig_of_cur.p, cur_of_orig.p, lo, num, m.seed,
                                                       list.p, info.p, colors.p);
        VSDMO_CHECK_LAUNCH();
        constexpr int CH = 4;
        ColourStatus h;
        for (long c0 = 0;; c0 += CH) {
            if (c0 > (long)num + CH) throw Error(VSDMO_E_CUDA, "colouring did not terminate");
            if (c0) VSDMO_CUDA(cudaMemsetAsync(cs.p->remaining, 0, sizeof(h.remaining), s));
            for (int i = 0; i < CH; ++i) {
                k_colour<<<(num + 255) / 256, 256, 0, s>>>(num, list.p, m.k - 1, info.p, first_fit, colors.p, cs.p->remaining + i,
                                                           i > 0 ? cs.p->remaining + i - 1 : nullptr, &cs.p->maxc,
                                                           cs.p->hist);
                VSDMO_CHECK_LAUNCH();
            }
            h = read_scalar(cs.p, s);
            if (h.remaining[CH - 1] == 0) break;
        }
        // the colours are dense: a first-fit colour k has neighbours of every colour below k, a round colour k
        // one of colour k - 1
        const int nc = h.maxc + 1;
        // stable sort of the range by colour
        DBuf<uint32_t> order(num, s);
        k_iota<<<G(num), 256, 0, s>>>(order.p, num);
        VSDMO_CHECK_LAUNCH();
        radix_sort_pairs((uint32_t*)colors.p, order.p, num, bits_for((uint32_t)(nc > 1 ? nc - 1 : 1)), s);
        offs_dev.alloc(nc + 1, s);
        if (nc <= 256) {
            k_colour_offsets<<<1, 256, 0, s>>>(cs.p->hist, nc, lo, offs_dev.p);
            VSDMO_CHECK_LAUNCH();
            offs_host.assign(1, lo);
            for (int c = 0; c < nc; ++c) offs_host.push_back(offs_host.back() + h.hist[c]);
        } else {
            rowptr_from_sorted((uint32_t*)colors.p, num, nc, offs_dev.p, s);
            k_add_const<<<G(nc + 1), 256, 0, s>>>(offs_dev.p, nc + 1, lo);
            VSDMO_CHECK_LAUNCH();
            offs_host = offs_dev.to_host();
        }
        permute_range((const int*)order.p, lo, num, flags);
        return nc;
    }

    // halfedges of the triangles / quads by source vertex; keys: the sources
    void halfedges(DBuf<uint32_t>& keys, DBuf<int>& rowptr, DBuf<int4>& he, int* longest) {
        const int nS = m.nSurf;
        const long n = (long)m.fk * m.nTris;
        DBuf<uint32_t> order(n, s);
        keys.alloc(n, s);
        VSDMO_CUDA(cudaMemcpyAsync(keys.p, m.tris.p, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
        rowptr.alloc(nS + 1, s);
        sort_short_rows(keys.p, order.p, n, nS, rowptr.p, longest, s);
        he.alloc(n, s);
        k_he_records<<<G(n), 256, 0, s>>>(order.p, n, m.tris.p, m.fk, he.p);
        VSDMO_CHECK_LAUNCH();
        k_opposite<<<G(n), 256, 0, s>>>(keys.p, he.p, n, rowptr.p, longest);
        VSDMO_CHECK_LAUNCH();
    }

    void surface_init() {
        const int nS = m.nSurf;
        const long nHE1 = (long)m.fk * m.nTris;
        m.fn.alloc(3L * m.nTris, s);
        k_face_normals<<<G(m.nTris), 256, 0, s>>>(m.tris.p, m.fk, m.nTris, m.pos.p, m.fn.p, at(&BuildStatus::surf_err));
        VSDMO_CHECK_LAUNCH();
        BuildStatus h;
        // first-pass halfedges; free vertices first, feature vertices last
        {
            DBuf<uint32_t> keys;
            DBuf<int> rowptr, order(nS, s);
            DBuf<int4> he;
            halfedges(keys, rowptr, he, at(&BuildStatus::longest_he));
            m.isB1.alloc(nS, s); m.isB1.zero();
            m.isFeat.alloc(nS, s); m.isFeat.zero();
            k_flags_b1_feat<<<G(nHE1), 256, 0, s>>>(keys.p, he.p, nHE1, m.fn.p, m.isB1.p, m.isFeat.p, m.isFlat,
                                                    at(&BuildStatus::nOpen), at(&BuildStatus::longest_he));
            VSDMO_CHECK_LAUNCH();
            if (m.isFlat) {
                k_copy_u8<<<G(nS), 256, 0, s>>>(m.isB1.p, m.isFeat.p, nS);
                VSDMO_CHECK_LAUNCH();
            }
            partition_flags(m.isFeat.p, nS, 0, order.p, at(&BuildStatus::nFree), s);
            h = status();
            check_err(h.surf_err, "surface");
            if (h.longest_he > SHORT_ROW_MAX) throw_long_fan();
            permute_range(order.p, 0, nS, {&m.isB1, &m.isFeat});
            m.nFeature = nS - h.nFree;
        }
        const int nFree = nS - m.nFeature;
        for (int part = 0; part < 2; ++part) {
            const int lo = part == 0 ? 0 : nFree, num = part == 0 ? nFree : m.nFeature;
            std::vector<int>& oh = part == 0 ? m.col_free : m.col_feature;
            DBuf<int>& od = part == 0 ? m.d_col_free : m.d_col_feature;
            int& nc = part == 0 ? m.nColFree : m.nColFeature;
            if (num <= 0) {
                oh.assign(1, lo);
                od.alloc(1, s);
                VSDMO_CUDA(cudaMemcpyAsync(od.p, oh.data(), sizeof(int), cudaMemcpyHostToDevice, s));
                nc = 0;
                continue;
            }
            nc = color_range(lo, num, oh, od, {&m.isB1, &m.isFeat});
        }
        final_halfedges(h.nOpen);
        m.vn.alloc(3L * nS, s);
        k_vertex_normals<<<G(nS), 256, 0, s>>>(nS, m.he_rowptr.p, m.he.p, m.fn.p, m.vn.p);
        VSDMO_CHECK_LAUNCH();
    }

    // nD: the boundary halfedges, each of which gets a dummy twin
    void final_halfedges(int nD) {
        const int nS = m.nSurf;
        const long nHE1 = (long)m.fk * m.nTris;
        DBuf<uint32_t> keys;
        DBuf<int> rowptr1;
        DBuf<int4> he1;
        halfedges(keys, rowptr1, he1, at(&BuildStatus::longest_he));
        DBuf<uint8_t> df(nHE1, s);
        k_dummy_flags<<<G(nHE1), 256, 0, s>>>(he1.p, nHE1, df.p);
        VSDMO_CHECK_LAUNCH();
        DBuf<int> didx(nHE1, s);
        compact_flags(df.p, nHE1, didx.p, nullptr, s);
        const long nHE = nHE1 + nD;
        DBuf<uint32_t> k2(nHE, s), o2(nHE, s);
        DBuf<int4> rec(nHE, s);
        k_with_dummies<<<G(nHE), 256, 0, s>>>(keys.p, he1.p, nHE1, didx.p, nD, k2.p, rec.p);
        VSDMO_CHECK_LAUNCH();
        m.he_rowptr.alloc(nS + 1, s);
        int* longest = at(&BuildStatus::longest_full);
        int* err = at(&BuildStatus::fan_err);
        sort_short_rows(k2.p, o2.p, nHE, nS, m.he_rowptr.p, longest, s);
        DBuf<int4> in(nHE, s);
        k_gather<int4><<<G(nHE), 256, 0, s>>>(rec.p, o2.p, in.p, nHE);
        VSDMO_CHECK_LAUNCH();
        k_opposite<<<G(nHE), 256, 0, s>>>(k2.p, in.p, nHE, m.he_rowptr.p, longest);
        VSDMO_CHECK_LAUNCH();
        m.he.alloc(nHE, s);
        k_ccw<<<G(nS), 256, 0, s>>>(nS, m.he_rowptr.p, in.p, m.he.p, m.isB1.p, m.isFeat.p, m.tris.p, m.fk, err, longest);
        VSDMO_CHECK_LAUNCH();
        k_opp_next<<<G(nS), 256, 0, s>>>(nS, m.he_rowptr.p, m.he.p, err, longest);
        VSDMO_CHECK_LAUNCH();
        const BuildStatus h = status();
        if (h.longest_full > SHORT_ROW_MAX) throw_long_fan();
        check_err(h.fan_err, "halfedges");
        m.maxHE = h.longest_full;
        m.nHE = (int)nHE;
    }

    // boundary triangles and boundary vertices of a tet mesh; the vertices' order, boundary first
    int tet_boundary(DBuf<int>& order) {
        const int nV = m.nV;
        const long nF = 4L * m.nE;
        DBuf<int> u(nV, s), offs((long)nV + 1, s);
        DBuf<unsigned long long> spill(nF, s);
        DBuf<uint8_t> spill_flag(nF, s);
        DBuf<ulonglong2> rec(nF, s);
        m.isB2.alloc(nV, s);
        m.isB2.zero();
        u.zero();
        k_tet_boundary<<<grid_for(32L * nV, FACE_WARPS * 32), FACE_WARPS * 32, 0, s>>>(
            inc_rs.p, inc.p, (const int4*)m.elems.p, nV, at(&BuildStatus::input_err), spill.p, spill_flag.p, at(&BuildStatus::spill), u.p,
            rec.p, at(&BuildStatus::nB), m.isB2.p, at(&BuildStatus::face_err), at(&BuildStatus::face_rows));
        VSDMO_CHECK_LAUNCH();
        exclusive_scan(u.p, offs.p, nV, offs.p + nV, s);
        order.alloc(nV, s);
        partition_flags(m.isB2.p, nV, 1, order.p, at(&BuildStatus::nS), s);
        const BuildStatus h = status();
        check_err(h.input_err, "input");
        if (h.face_rows > SHORT_ROW_MAX)
            throw Error(VSDMO_E_VALENCE, "a vertex is the first corner of more than " + std::to_string(SHORT_ROW_MAX) +
                                             " tetrahedron faces (more than ~1365 tetrahedra around one vertex)");
        check_err(h.face_err, "boundary faces");
        m.nTris = h.nB;
        m.tris.alloc(3L * h.nB, s);
        k_face_emit<<<G(h.nB), 256, 0, s>>>(rec.p, h.nB, offs.p, m.tris.p);
        VSDMO_CHECK_LAUNCH();
        order_elem_rows(h);
        return h.nS;
    }

    // the rows of the vertex-to-element table longer than one warp orders (the others are)
    void order_elem_rows(const BuildStatus& h) {
        m.maxTets = h.longest_elems;
        if (h.longest_elems > SHORT_ROW_MAX) sort_long_rows((const uint32_t*)m.elems.p, inc.p, (long)inc.n, m.nV, s);
    }

    void hex_boundary() {
        const int nH = m.nE;
        const long nF = 6L * nH;
        DBuf<uint32_t> f0(nF, s), f1(nF, s), f2(nF, s), f3(nF, s), key(nF, s), order(nF, s);
        k_hex_faces<<<G(nH), 256, 0, s>>>(m.elems.p, nH, f0.p, f1.p, f2.p, f3.p);
        VSDMO_CHECK_LAUNCH();
        k_iota<<<G(nF), 256, 0, s>>>(order.p, nF);
        VSDMO_CHECK_LAUNCH();
        const int bits = bits_for((uint32_t)(m.nV - 1));
        const uint32_t* comps[4] = { f3.p, f2.p, f1.p, f0.p };
        for (int c = 0; c < 4; ++c) {
            k_gather_key<<<G(nF), 256, 0, s>>>(comps[c], order.p, key.p, nF);
            VSDMO_CHECK_LAUNCH();
            radix_sort_pairs(key.p, order.p, nF, bits, s);
        }
        DBuf<uint32_t> s0(nF, s), s1(nF, s), s2(nF, s), s3(nF, s);
        k_gather_key<<<G(nF), 256, 0, s>>>(f0.p, order.p, s0.p, nF);
        k_gather_key<<<G(nF), 256, 0, s>>>(f1.p, order.p, s1.p, nF);
        k_gather_key<<<G(nF), 256, 0, s>>>(f2.p, order.p, s2.p, nF);
        k_gather_key<<<G(nF), 256, 0, s>>>(f3.p, order.p, s3.p, nF);
        VSDMO_CHECK_LAUNCH();
        DBuf<uint8_t> paired(nF, s), unpaired(nF, s);
        paired.zero();
        k_pair_quads<<<G(nF), 256, 0, s>>>(s0.p, s1.p, s2.p, s3.p, nF, paired.p, at(&BuildStatus::face_err));
        VSDMO_CHECK_LAUNCH();
        k_not<<<G(nF), 256, 0, s>>>(paired.p, unpaired.p, nF);
        VSDMO_CHECK_LAUNCH();
        DBuf<int> bidx(nF, s);
        compact_flags(unpaired.p, nF, bidx.p, at(&BuildStatus::nB), s);
        const BuildStatus h = status();
        check_err(h.face_err, "boundary faces");
        const int nB = h.nB;
        m.nTris = nB;
        m.tris.alloc(4L * nB, s);
        m.isB2.alloc(m.nV, s);
        m.isB2.zero();
        k_emit_boundary_quads<<<G(nB), 256, 0, s>>>(bidx.p, nB, s0.p, s1.p, s2.p, s3.p, m.tris.p, m.isB2.p);
        VSDMO_CHECK_LAUNCH();
        order_elem_rows(h);
    }

    // the elements in the final vertex numbering and the halffaces / halfhexes, rows in element order
    void finish_elems() {
        const long n = (long)m.k * m.nE;
        k_remap<<<G(n), 256, 0, s>>>(m.elems.p, n, cur_of_orig.p);
        VSDMO_CHECK_LAUNCH();
        m.hf_rowptr.alloc(m.nV + 1, s);
        DBuf<int> len(m.nV, s);
        k_row_lengths<<<G(m.nV), 256, 0, s>>>(inc_rs.p, orig_of_cur.p, m.nV, len.p);
        VSDMO_CHECK_LAUNCH();
        exclusive_scan(len.p, m.hf_rowptr.p, m.nV, m.hf_rowptr.p + m.nV, s);
        if (m.type == VSDMO_HEX) {
            m.hh.alloc(2 * n, s);
            k_halfhexes<<<G(8L * m.nV), 256, 0, s>>>(inc_rs.p, inc.p, orig_of_cur.p, m.hf_rowptr.p, m.nV, m.elems.p, m.hh.p);
        } else {
            m.hf.alloc(n, s);
            k_halffaces<<<G(8L * m.nV), 256, 0, s>>>(inc_rs.p, inc.p, orig_of_cur.p, m.hf_rowptr.p, m.nV,
                                                     (const int4*)m.elems.p, m.hf.p);
        }
        VSDMO_CHECK_LAUNCH();
    }

    // boundary vertices first, the inner ones coloured and sorted, then the surface
    void volume(const int* order, int nS) {
        permute_range(order, 0, m.nV, {&m.isB2});
        m.nSurf = nS;
        const int nI = m.nV - nS;
        if (nI > 0) {
            m.nColInner = color_range(nS, nI, m.col_inner, m.d_col_inner, {&m.isB2});
        } else {
            m.nColInner = 0;
            m.col_inner.assign(1, nS);
            m.d_col_inner.alloc(1, s);
            VSDMO_CUDA(cudaMemcpyAsync(m.d_col_inner.p, m.col_inner.data(), sizeof(int), cudaMemcpyHostToDevice, s));
        }
        if (nS > 0) surface_init();
        finish_elems();
    }

    void run(const float* d_xyz, const int* d_elems) {
        const long nIdx = (long)m.nE * m.k;
        m.pos.alloc(m.nV, s);
        m.elems.alloc(nIdx, s);
        orig_of_cur.alloc(m.nV, s);
        cur_of_orig.alloc(m.nV, s);
        st.alloc(1, s);
        st.zero();
        const bool volume_mesh = m.type != VSDMO_TRI && m.type != VSDMO_QUAD;
        inc_rs.alloc((long)m.nV + 1, s);
        inc.alloc(nIdx, s);
        {
            DBuf<int> counts(m.nV, s), slot(nIdx, s);
            counts.zero();
            k_input<<<G(std::max<long>(m.nV, nIdx)), 256, 0, s>>>(d_xyz, m.nV, d_elems, nIdx, m.pos.p, orig_of_cur.p, cur_of_orig.p,
                                                                  m.elems.p, counts.p, slot.p, at(&BuildStatus::input_err),
                                                                  at(&BuildStatus::nonzero_z));
            VSDMO_CHECK_LAUNCH();
            if (volume_mesh) {
                DBuf<uint32_t> rows(nIdx, s);
                rows_from_slots((const uint32_t*)m.elems.p, slot.p, counts.p, nIdx, m.nV, inc_rs.p, rows.p, s);
                order_short_rows(inc_rs.p, rows.p, m.nV, inc.p, nullptr, at(&BuildStatus::longest_elems), s);
            } else {
                rows_from_slots((const uint32_t*)m.elems.p, slot.p, counts.p, nIdx, m.nV, inc_rs.p, inc.p, s);
            }
        }
        if (!volume_mesh) {
            const BuildStatus h = status();
            check_err(h.input_err, "input");
            m.fk = m.k;
            m.isFlat = h.nonzero_z ? 0 : 1;
            m.nSurf = m.nV;
            m.nTris = m.nE;
            m.tris.alloc(nIdx, s);
            VSDMO_CUDA(cudaMemcpyAsync(m.tris.p, m.elems.p, sizeof(int) * nIdx, cudaMemcpyDeviceToDevice, s));
            m.col_inner.assign(1, m.nV);
            m.d_col_inner.alloc(1, s);
            VSDMO_CUDA(cudaMemcpyAsync(m.d_col_inner.p, m.col_inner.data(), sizeof(int), cudaMemcpyHostToDevice, s));
            surface_init();
            VSDMO_CUDA(cudaMemcpyAsync(m.elems.p, m.tris.p, sizeof(int) * nIdx, cudaMemcpyDeviceToDevice, s));
        } else if (m.type == VSDMO_TET) {
            m.fk = 3;
            m.isFlat = 0;
            DBuf<int> order;
            const int nS = tet_boundary(order);
            volume(order.p, nS);
        } else {  // VSDMO_HEX (MeshHexGPU::init, mesh/MeshHexGPU.cu:35-43)
            m.fk = 4;
            m.isFlat = 0;
            check_err(status().input_err, "input");
            hex_boundary();
            DBuf<int> order(m.nV, s);
            partition_flags(m.isB2.p, m.nV, 1, order.p, at(&BuildStatus::nS), s);
            volume(order.p, status().nS);
        }
        m.new_of_old = std::move(cur_of_orig);
        m.sync();
    }
};

}  // namespace

void build_mesh(Mesh& m, const float* d_xyz, const int* d_elems) {
    Builder b(m);
    b.run(d_xyz, d_elems);
}

void update_normals(const Mesh& m, cudaStream_t s) {
    if (m.nTris <= 0 || m.nSurf <= 0) return;
    k_face_normals<<<G(m.nTris), 256, 0, s>>>(m.tris.p, m.fk, m.nTris, m.pos.p, m.fn.p, nullptr);
    VSDMO_CHECK_LAUNCH();
    k_vertex_normals<<<G(m.nSurf), 256, 0, s>>>(m.nSurf, m.he_rowptr.p, m.he.p, m.fn.p, m.vn.p);
    VSDMO_CHECK_LAUNCH();
}

}  // namespace vsdmo
