// fuzzy.cu -- the fuzzy simplicial set on the device (src/fuzzy.rs:25-91):
// the symmetrized membership graph that consumes the kNN graph and its
// calibration, as COO sorted by (row, col).
//
// Row r of the output is the sorted union of two lists: F_r, the columns of
// row r's own kNN list with a nonzero directed strength A[r][c], and R_r,
// the rows s whose lists hold r with A[s][r] nonzero.  Each is a set (the
// indices of a row are distinct), so
//
//   1. fuzzy_entries_kernel (one thread per kNN entry) computes the strengths
//      (self skipped; 1 when d - rho <= 0 or sigma == 0, else libm
//      expf(-(d / sigma)); zeros dropped) and counts each column's arrivals:
//      the count returned is the entry's slot in R_col.
//   2. fuzzy_segments_kernel gives every row a segment of k + |R_r| slots (in
//      any order: one atomic per block).
//   3. fuzzy_scatter_kernel drops (source, strength) into R_r's slots.
//   4. fuzzy_union_kernel (one warp per row of at most 128 slots) sorts the
//      row's F and R entries in registers, forms the binary32 t-conorm
//      (v + vt) - v * vt of equal columns in the reference's order
//      (src/fuzzy.rs:67-75) and leaves the sorted row at the front of its
//      segment; fuzzy_long_kernel does the rows above 128 slots: a warp each up
//      to 512, a block each beyond, several to one of very many arrivals.
//   5. fuzzy_write_kernel (one block per tile of rows, several per very long row)
//      sums the tiles before it, scans its rows' counts and writes the COO.
//
// Strengths lie in [0, 1] (or are NaN) when every sigma is non-negative, and
// then no fused value of a union coordinate is zero: fl(v * vt) <= min(v,
// vt) <= max(v, vt) <= fl(v + vt) with one of the inequalities strict, so
// the difference is positive.  The reference's zero filter after the fusion
// therefore drops nothing and the union size is the entry count.  The slots
// depend on the order of the atomics, the sorted rows do not: the output is
// the reference's, entry for entry.
//
// What bounds it: latency of the L2-resident arrays and the sorts' issue.  With a
// radix sort of the reverse copies and binary-search merges -> now: kNN graph of
// 50,000 x 384 embeddings, k = 30 (2.7 M entries) 183 -> 110 us; random graphs of
// 100,000 x 15 250 -> 104, 2,000 x 15 60 -> 28.
#include <cuda_runtime.h>

#include <algorithm>

#include "hm_internal.cuh"
#include "libm_expf.cuh"

namespace hm {

constexpr unsigned FZ_FULL = 0xffffffffu;
// bits of the status word for inputs outside the precondition (each row's
// indices distinct and below n)
constexpr uint32_t FZ_BAD_INDEX = 1u, FZ_BAD_DUPLICATE = 2u;
constexpr uint32_t FZ_SLOT_BITS = 9;                     // slots of a warp-sorted row: 512
constexpr uint32_t FZ_WARP_SLOTS = 1u << FZ_SLOT_BITS;
constexpr uint32_t FZ_SHORT_SLOTS = 128;                 // and of the short-row kernel
constexpr uint32_t FZ_TILES = 1024;                      // write tiles at most
constexpr uint32_t FZ_TILE_ROWS = 32;                    // and rows per tile at least
constexpr uint32_t FZ_WINDOW = 1u << 19;                 // columns per pass of the hub kernel
constexpr uint32_t FZ_PART_WINDOW = 1u << 14;            // and where several blocks share a hub
constexpr uint32_t FZ_SHARED_HUB = 8192;                 // of this many arrivals
constexpr uint32_t FZ_HOT = 8;                           // matches that make a block of entries count jointly
constexpr uint32_t FZ_JOINT_ROWS = 2048;                 // in graphs of this many rows
enum { FZ_ALLOCATED = 0, FZ_HUBS = 1, FZ_BAD = 2, FZ_MIDS = 3, FZ_NEXT = 4, FZ_WORDS = 8 };

struct FuzzyDev {
    const uint32_t *idx;
    const float *dist, *sigma, *rho;
    uint32_t n, k, entries, tile_rows;
    float *w;           // directed strengths (0: dropped)
    uint32_t *slot;     // slot of the entry in its column's R list
    uint32_t *indeg;    // |R_r|
    uint32_t *seg;      // first slot of row r's segment
    uint2 *stage;       // segments: (source or column, strength bits)
    uint2 *hub_out;     // rows of more than 512 slots, at their segments' places
    uint32_t *count;    // entries of output row r
    uint32_t *tile_sum;
    uint32_t *longs;    // rows of more than 512 slots from the front, of 129 to 512 from the back (mid_row)
    uint32_t *words;    // FZ_*
};

__device__ __forceinline__ uint32_t &mid_row(const FuzzyDev &D, uint32_t i) { return D.longs[D.n - 1 - i]; }

__device__ __forceinline__ float tconorm(float v, float vt) {
    return __fsub_rn(__fadd_rn(v, vt), __fmul_rn(v, vt));
}

constexpr uint32_t FZ_PER_THREAD = 4;  // entries in flight per thread of the entry kernels

// Arrival slots of a block's 256 * FZ_PER_THREAD entries whose rows list the same
// columns at the same places (points at distance 0 from all, such as zero vectors
// under cosine): a column's counter would take an atomic from every row.  The warps
// go down the places instead, 32 rows at a time, and equal columns share one.
// col[e]: the column of the block's entry e, or ~0u; receives its slot.
__device__ __noinline__ void joint_slots(const FuzzyDev &D, uint32_t *col) {
    constexpr uint32_t N = 256 * FZ_PER_THREAD;
    const uint32_t lane = threadIdx.x & 31, k = min(D.k, N), rows = (N + k - 1) / k;
    for (uint32_t t0 = 0; t0 < k * rows; t0 += 256) {  // whole warps
        const uint32_t t = t0 + threadIdx.x, e = (t % rows) * k + t / rows;
        const bool in = t < k * rows && e < N;
        const uint32_t c = in ? col[e] : ~0u;
        const unsigned m = __match_any_sync(FZ_FULL, c);
        const int leader = __ffs(m) - 1;
        uint32_t base = 0;
        if (c != ~0u && (int)lane == leader) base = atomicAdd(&D.indeg[c], (uint32_t)__popc(m));
        base = __shfl_sync(FZ_FULL, base, leader);
        if (in) col[e] = base + __popc(m & ((1u << lane) - 1u));
    }
}

__global__ void __launch_bounds__(256) fuzzy_entries_kernel(const FuzzyDev D) {
    __shared__ uint32_t s_col[256 * FZ_PER_THREAD];
    grid_ready();
    const uint32_t e0 = blockIdx.x * 256 * FZ_PER_THREAD + threadIdx.x;
    uint32_t col[FZ_PER_THREAD], row[FZ_PER_THREAD], slot[FZ_PER_THREAD];
    float d[FZ_PER_THREAD], sg[FZ_PER_THREAD], w[FZ_PER_THREAD];
#pragma unroll
    for (uint32_t q = 0; q < FZ_PER_THREAD; ++q) {
        const uint32_t e = min(e0 + 256 * q, D.entries - 1);
        row[q] = e / D.k;
        col[q] = D.idx[e];
        d[q] = __fsub_rn(D.dist[e], D.rho[row[q]]);
        sg[q] = D.sigma[row[q]];
    }
    const bool same = D.n >= FZ_JOINT_ROWS && e0 + D.k < D.entries && D.idx[e0 + D.k] == col[0];
#pragma unroll
    for (uint32_t q = 0; q < FZ_PER_THREAD; ++q) {
        w[q] = 0.0f;
        slot[q] = 0;
        if (e0 + 256 * q >= D.entries) continue;
        if (col[q] >= D.n) {
            // outside the precondition: dropped (so every later index stays in
            // bounds) and reported through the status word
            atomicOr(&D.words[FZ_BAD], FZ_BAD_INDEX);
        } else if (col[q] != row[q]) {
            if (!(d[q] <= 0.0f || sg[q] == 0.0f)) {
                const float x = -__fdiv_rn(d[q], sg[q]);
                w[q] = x <= 0.0f ? expf_libm_nonpos(x) : expf_libm(x);
            } else {
                w[q] = 1.0f;
            }
        }
    }
    // whether rows list the same columns at the same places: a quarter of the block's
    // entries against the row below (FZ_HOT of 256: one shared column in 30).  A counter
    // takes an atomic in 2.5 ns, so small graphs gain nothing (100 x 50: 25 us, 27 if
    // counted jointly).
    const bool joint = D.n >= FZ_JOINT_ROWS && __syncthreads_count(same) >= FZ_HOT;
    if (!joint) {
#pragma unroll
        for (uint32_t q = 0; q < FZ_PER_THREAD; ++q)
            if (w[q] != 0.0f) slot[q] = atomicAdd(&D.indeg[col[q]], 1u);
    } else {
#pragma unroll
        for (uint32_t q = 0; q < FZ_PER_THREAD; ++q) s_col[256 * q + threadIdx.x] = w[q] != 0.0f ? col[q] : ~0u;
        __syncthreads();
        joint_slots(D, s_col);
        __syncthreads();
#pragma unroll
        for (uint32_t q = 0; q < FZ_PER_THREAD; ++q) slot[q] = s_col[256 * q + threadIdx.x];
    }
#pragma unroll
    for (uint32_t q = 0; q < FZ_PER_THREAD; ++q) {
        if (e0 + 256 * q >= D.entries) continue;
        D.w[e0 + 256 * q] = w[q];
        D.slot[e0 + 256 * q] = slot[q];
    }
}

// inclusive scan of v over the warp
__device__ __forceinline__ uint32_t warp_scan(uint32_t v, uint32_t lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FZ_FULL, v, o);
        if (lane >= (uint32_t)o) v += y;
    }
    return v;
}
// exclusive scan of v over a block of 256 threads, its total in `sum`
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t *warp_sums, uint32_t &sum) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t incl = warp_scan(v, lane);
    __syncthreads();
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    uint32_t before = 0;
    sum = 0;
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) {
        before += q < warp ? warp_sums[q] : 0u;
        sum += warp_sums[q];
    }
    return before + incl - v;
}

__global__ void __launch_bounds__(256) fuzzy_segments_kernel(const FuzzyDev D) {
    grid_ready();
    __shared__ uint32_t warp_sums[8], base;
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t mine = r < D.n ? D.k + D.indeg[r] : 0u;
    uint32_t sum;
    const uint32_t at = block_scan(mine, warp_sums, sum);
    if (threadIdx.x == 0) base = atomicAdd(&D.words[FZ_ALLOCATED], sum);
    __syncthreads();
    if (r < D.n) D.seg[r] = base + at;
}

__global__ void __launch_bounds__(256) fuzzy_scatter_kernel(const FuzzyDev D) {
    grid_ready();
    const uint32_t e0 = blockIdx.x * 256 * FZ_PER_THREAD + threadIdx.x;
    float w[FZ_PER_THREAD];
    uint32_t at[FZ_PER_THREAD];
#pragma unroll
    for (uint32_t q = 0; q < FZ_PER_THREAD; ++q) {
        const uint32_t e = min(e0 + 256 * q, D.entries - 1);
        w[q] = e0 + 256 * q < D.entries ? D.w[e] : 0.0f;
        at[q] = (w[q] != 0.0f ? D.seg[D.idx[e]] : 0u) + D.k + D.slot[e];
    }
#pragma unroll
    for (uint32_t q = 0; q < FZ_PER_THREAD; ++q)
        if (w[q] != 0.0f && at[q] < 2 * D.entries) D.stage[at[q]] = make_uint2((e0 + 256 * q) / D.k, __float_as_uint(w[q]));
}

// A row of at most 32 * NQ slots: keys column << 9 | slot (F slots below k, so an
// F entry precedes its R partner), strengths in shared memory by slot.
template <typename K, int NQ>
__device__ __forceinline__ uint32_t union_row(const FuzzyDev &D, uint32_t r, uint32_t slots, float *w, uint32_t lane) {
    const uint32_t k = D.k;
    const uint64_t base = (uint64_t)r * k;
    uint2 *seg = D.stage + D.seg[r];
    K v[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const uint32_t e = q * 32 + lane;
        v[q] = ~(K)0;
        if (e < k) {
            const float f = D.w[base + e];
            if (f != 0.0f) v[q] = (K)D.idx[base + e] << FZ_SLOT_BITS | e;
            w[e] = f;
        } else if (e < slots) {
            const uint2 s = seg[e];
            v[q] = (K)s.x << FZ_SLOT_BITS | e;
            w[e] = __uint_as_float(s.y);
        }
    }
    warp_sort<K, NQ>(v, lane);
    __syncwarp();  // w, and every read of the segment before its first write
    const K before = __shfl_up_sync(FZ_FULL, v[NQ - 1], 1), after = __shfl_down_sync(FZ_FULL, v[0], 1);
    auto col = [](K key) { return key >> FZ_SLOT_BITS; };
    uint32_t keep = 0;
    bool dup = false;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const bool first = q == 0 && lane == 0;
        const K prev = q == 0 ? before : v[q - 1];
        const bool same = !first && col(prev) == col(v[q]);
        if (v[q] != ~(K)0) {
            if (!same) keep |= 1u << q;
            else dup |= ((uint32_t)v[q] & (FZ_WARP_SLOTS - 1)) < k;  // an F entry after another
        }
    }
    if (dup) atomicOr(&D.words[FZ_BAD], FZ_BAD_DUPLICATE);
    const uint32_t mine = __popc(keep), incl = warp_scan(mine, lane);
    uint32_t at = incl - mine;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        if (!(keep >> q & 1u)) continue;
        const K next = q == NQ - 1 ? after : v[q + 1];
        const bool last = q == NQ - 1 && lane == 31;
        const uint32_t slot = (uint32_t)v[q] & (FZ_WARP_SLOTS - 1);
        const float own = w[slot];
        const bool pair = !last && next != ~(K)0 && col(next) == col(v[q]);
        const float other = pair ? w[(uint32_t)next & (FZ_WARP_SLOTS - 1)] : 0.0f;
        const float f = slot < k ? tconorm(own, other) : tconorm(0.0f, own);
        seg[at++] = make_uint2((uint32_t)col(v[q]), __float_as_uint(f));
    }
    return __shfl_sync(FZ_FULL, incl, 31);
}

// Rows of at most 128 slots (nine in ten at k = 30), one warp each; the others go
// to the lists of the next kernel, which keeps this one at 32 registers and its
// blocks even.
constexpr int FZ_WARPS = 4;
template <typename K>
__global__ void __launch_bounds__(FZ_WARPS * 32, sizeof(K) == 4 ? 16 : 8) fuzzy_union_kernel(const FuzzyDev D) {
    grid_ready();
    __shared__ float w_all[FZ_WARPS][FZ_SHORT_SLOTS];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t r = blockIdx.x * FZ_WARPS + warp;
    if (r >= D.n) return;  // whole warps
    const uint32_t slots = D.k + D.indeg[r];
    uint32_t count;
    if (slots <= 64) count = union_row<K, 2>(D, r, slots, w_all[warp], lane);
    else if (slots <= FZ_SHORT_SLOTS) count = union_row<K, 4>(D, r, slots, w_all[warp], lane);
    else {
        if (lane == 0) {
            if (D.n + D.k <= FZ_SHORT_SLOTS) {
                // (no long-row kernel follows: distinct indices give a row k slots and
                // at most n - 1 arrivals, so an index is repeated)
                atomicOr(&D.words[FZ_BAD], FZ_BAD_DUPLICATE);
                D.count[r] = 0;
            } else if (slots <= FZ_WARP_SLOTS) {
                mid_row(D, atomicAdd(&D.words[FZ_MIDS], 1u)) = r;
            } else {
                D.longs[atomicAdd(&D.words[FZ_HUBS], 1u)] = r;
            }
        }
        return;
    }
    if (lane == 0) {
        D.count[r] = count;
        atomicAdd(&D.tile_sum[r / D.tile_rows], count);
    }
}

// The block's columns [c0, c0 + width) of a hub row, for one of several blocks that
// share it.  One pass over the arrivals counts those below the window and leaves the
// others' strengths by column; with the F entries below the window less those that
// arrived too (found in the lists of their own rows), that is where the window starts
// in the row.  smem: width strengths, then three words per 32 columns.
__device__ __forceinline__ void hub_part(const FuzzyDev &D, uint32_t r, uint32_t c0, uint32_t width, uint32_t *smem,
                                         uint32_t *warp_sums) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, k = D.k;
    const uint32_t c1 = min(D.n - c0, width), nw = (c1 + 31) / 32;  // the window's columns, words (at most 1,024)
    uint32_t *strength = smem, *rbits = strength + width, *fbits = rbits + (width + 31) / 32, *pre = fbits + (width + 31) / 32;
    const uint32_t rc = D.indeg[r];
    const uint64_t base = (uint64_t)r * k;
    const uint2 *seg = D.stage + D.seg[r];
    uint2 *out = D.hub_out + D.seg[r];
    __shared__ uint32_t s_below;
    __syncthreads();
    if (tid < nw) rbits[tid] = fbits[tid] = 0u;
    if (tid == 0) s_below = 0;
    __syncthreads();
    uint32_t below = 0;
    for (uint32_t e = tid; e < rc; e += 8 * 1024) {
        uint2 s[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) s[q] = e + 1024 * q < rc ? seg[k + e + 1024 * q] : make_uint2(~0u, 0u);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const uint32_t c = s[q].x - c0;
            below += s[q].x < c0 ? 1u : 0u;
            if (s[q].x >= c0 && c < c1) {
                atomicOr(&rbits[c >> 5], 1u << (c & 31));
                strength[c] = s[q].y;
            }
        }
    }
    for (uint32_t e = warp; e < k; e += 32) {  // a warp per F entry
        const uint32_t col = D.idx[base + e];
        if (D.w[base + e] == 0.0f) continue;
        if (col < c0) {
            const uint64_t other = (uint64_t)col * k;
            bool partner = false;
            for (uint32_t j = lane; j < k; j += 32) partner |= D.idx[other + j] == r && D.w[other + j] != 0.0f;
            if (!__any_sync(FZ_FULL, partner) && lane == 0) ++below;
        } else if (col - c0 < c1 && lane == 0) {
            const uint32_t c = col - c0, bit = 1u << (c & 31);
            if (atomicOr(&fbits[c >> 5], bit) & bit) atomicOr(&D.words[FZ_BAD], FZ_BAD_DUPLICATE);
        }
    }
    below = __reduce_add_sync(FZ_FULL, below);
    if (lane == 0 && below) atomicAdd(&s_below, below);
    __syncthreads();
    const uint32_t v = tid < nw ? __popc(rbits[tid] | fbits[tid]) : 0u, incl = warp_scan(v, lane);
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    const uint32_t ws = warp_scan(warp_sums[lane], lane);
    const uint32_t before = __shfl_sync(FZ_FULL, ws, warp ? warp - 1 : 0), sum = __shfl_sync(FZ_FULL, ws, 31);
    const uint32_t start = s_below;
    if (tid < nw) pre[tid] = start + (warp ? before : 0u) + incl - v;
    __syncthreads();
    auto place = [&](uint32_t c) {
        const uint32_t q = c >> 5;
        return pre[q] + __popc((rbits[q] | fbits[q]) & ((1u << (c & 31)) - 1u));
    };
    for (uint32_t c = tid; c < c1; c += 1024)  // R entries without an F partner
        if ((rbits[c >> 5] & ~fbits[c >> 5]) >> (c & 31) & 1u)
            out[place(c)] = make_uint2(c0 + c, __float_as_uint(tconorm(0.0f, __uint_as_float(strength[c]))));
    for (uint32_t e = tid; e < k; e += 1024) {
        const uint32_t col = D.idx[base + e], c = col - c0;
        const float f = D.w[base + e];
        if (f == 0.0f || col < c0 || c >= c1) continue;
        const float vt = rbits[c >> 5] >> (c & 31) & 1u ? __uint_as_float(strength[c]) : 0.0f;
        out[place(c)] = make_uint2(col, __float_as_uint(tconorm(f, vt)));
    }
    if (tid == 0 && c0 + c1 == D.n) {
        D.count[r] = start + sum;
        atomicAdd(&D.tile_sum[r / D.tile_rows], start + sum);
    }
}

// Rows of more than 512 slots (hubs): R_r and F_r as bitmaps over the columns, whose
// prefix counts give every entry's place with no sort.  Zero vectors under cosine are
// at distance 0 from every point, so rows with n entries do occur, and then there are
// few of them: where the blocks are at least twice the hubs, each long hub is shared
// by several (hub_part); else a block takes hubs in turn, windows of 2^19 columns at a
// time.  (Sharing hubs of 600 arrivals as well keeps all blocks from the other rows:
// the embeddings' graph above 105 -> 112 us.)  The rows are built beside the segments,
// which every window reads.
// The blocks' warps then take the rows of 129 to 512 slots, one each.
// Graphs whose rows share their neighbours, one block a hub and an atomic an entry ->
// now (both kernels): 50,000 x 30 with 29 shared 260 -> 110 us, 200,000 x 15 with 14
// 656 -> 270, with one 530 -> 236; sorting the arrivals took 141, 335 and 447.
template <typename K>
__global__ void __launch_bounds__(1024) fuzzy_long_kernel(const FuzzyDev D) {
    grid_ready();
    extern __shared__ uint32_t hub_smem[];
    __shared__ uint32_t warp_sums[32];
    const uint32_t words_n = (min(D.n, FZ_WINDOW) + 31) / 32;
    uint32_t *rbits = hub_smem, *fbits = rbits + words_n, *pre = fbits + words_n;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t hubs = D.words[FZ_HUBS], k = D.k, parts = hubs ? gridDim.x / hubs : 0u;
    const bool spread = parts > 1;  // the blocks of hub h: h parts, ..., h parts + parts - 1
    for (uint32_t h = spread ? blockIdx.x / parts : blockIdx.x; h < hubs; h += spread ? hubs : gridDim.x) {
        const uint32_t r = D.longs[h], rc = D.indeg[r];
        if (spread && rc >= FZ_SHARED_HUB) {
            const uint32_t width = min(((D.n + parts - 1) / parts + 31) & ~31u, FZ_PART_WINDOW);
            for (uint64_t c0 = (uint64_t)(blockIdx.x % parts) * width; c0 < D.n; c0 += (uint64_t)parts * width)
                hub_part(D, r, (uint32_t)c0, width, hub_smem, warp_sums);
            continue;
        }
        if (spread && blockIdx.x % parts) continue;
        const uint64_t base = (uint64_t)r * k;
        const uint2 *seg = D.stage + D.seg[r];
        uint2 *out = D.hub_out + D.seg[r];
        uint32_t total = 0;
        for (uint32_t c0 = 0; c0 < D.n; c0 += FZ_WINDOW) {
            const uint32_t c1 = min(D.n - c0, FZ_WINDOW), nw = (c1 + 31) / 32;  // the window's columns, words
            __syncthreads();
            for (uint32_t q = tid; q < nw; q += 1024) rbits[q] = fbits[q] = 0u;
            __syncthreads();
            for (uint32_t e = tid; e < rc; e += 8 * 1024) {  // eight loads in flight: n arrivals, one block
                uint32_t c[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) c[q] = e + 1024 * q < rc ? seg[k + e + 1024 * q].x - c0 : ~0u;
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (c[q] < c1) atomicOr(&rbits[c[q] >> 5], 1u << (c[q] & 31));
            }
            for (uint32_t e = tid; e < k; e += 1024) {
                const uint32_t c = D.idx[base + e] - c0, bit = 1u << (c & 31);
                if (D.w[base + e] != 0.0f && c < c1 && (atomicOr(&fbits[c >> 5], bit) & bit))
                    atomicOr(&D.words[FZ_BAD], FZ_BAD_DUPLICATE);
            }
            __syncthreads();
            uint32_t carry = total;
            for (uint32_t q0 = 0; q0 < nw; q0 += 1024) {
                const uint32_t q = q0 + tid, v = q < nw ? __popc(rbits[q] | fbits[q]) : 0u;
                const uint32_t incl = warp_scan(v, lane);
                if (lane == 31) warp_sums[warp] = incl;
                __syncthreads();
                const uint32_t ws = warp_scan(warp_sums[lane], lane);
                const uint32_t before = __shfl_sync(FZ_FULL, ws, warp ? warp - 1 : 0);
                if (q < nw) pre[q] = carry + (warp ? before : 0u) + incl - v;
                carry += __shfl_sync(FZ_FULL, ws, 31);
                __syncthreads();
            }
            auto place = [&](uint32_t c) {
                const uint32_t q = c >> 5;
                return pre[q] + __popc((rbits[q] | fbits[q]) & ((1u << (c & 31)) - 1u));
            };
            // R entries; one with an F partner leaves its strength for it
            for (uint32_t e = tid; e < rc; e += 4 * 1024) {
                uint2 s[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) s[q] = e + 1024 * q < rc ? seg[k + e + 1024 * q] : make_uint2(~0u, 0u);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t c = s[q].x - c0;
                    if (e + 1024 * q >= rc || c >= c1) continue;
                    const bool partner = fbits[c >> 5] >> (c & 31) & 1u;
                    out[place(c)] = make_uint2(
                        s[q].x, partner ? s[q].y : __float_as_uint(tconorm(0.0f, __uint_as_float(s[q].y))));
                }
            }
            __syncthreads();
            for (uint32_t e = tid; e < k; e += 1024) {
                const uint32_t col = D.idx[base + e], c = col - c0;
                const float v = D.w[base + e];
                if (v == 0.0f || c >= c1) continue;
                const uint32_t at = place(c);
                const float vt = rbits[c >> 5] >> (c & 31) & 1u ? __uint_as_float(out[at].y) : 0.0f;
                out[at] = make_uint2(col, __float_as_uint(tconorm(v, vt)));
            }
            total = carry;
        }
        if (tid == 0) {
            D.count[r] = total;
            atomicAdd(&D.tile_sum[r / D.tile_rows], total);
        }
    }
    __syncthreads();
    float *w = reinterpret_cast<float *>(hub_smem) + warp * FZ_WARP_SLOTS;
    const uint32_t mids = D.words[FZ_MIDS];
    for (;;) {  // taken as warps come free: blocks without hubs take most
        uint32_t i = lane == 0 ? atomicAdd(&D.words[FZ_NEXT], 1u) : 0u;
        i = __shfl_sync(FZ_FULL, i, 0);
        if (i >= mids) break;
        const uint32_t r = mid_row(D, i), slots = k + D.indeg[r];
        const uint32_t count = slots <= 256 ? union_row<K, 8>(D, r, slots, w, lane) : union_row<K, 16>(D, r, slots, w, lane);
        __syncwarp();
        if (lane == 0) {
            D.count[r] = count;
            atomicAdd(&D.tile_sum[r / D.tile_rows], count);
        }
    }
}

// Entries of the tiles before `tile` (a whole block).
__device__ __forceinline__ uint32_t tile_offset(const FuzzyDev &D, uint32_t tile, uint32_t *warp_sums) {
    uint32_t sum = 0, total;
    for (uint32_t t = threadIdx.x; t < tile; t += 256) sum += D.tile_sum[t];
    block_scan(sum, warp_sums, total);
    return total;
}

// The COO: a block per tile of tile_rows rows, its warps taking the rows in turn.  Hub
// rows of more than 512 entries are left to the blocks past the tiles, several to a
// row, unless there are more such rows than blocks.  (Every offset lies below 2 n k;
// the comparisons keep a kernel that was handed something else in its arrays.)
__global__ void __launch_bounds__(256) fuzzy_write_kernel(const FuzzyDev D, uint32_t tiles, uint32_t *__restrict__ rows,
                                                          uint32_t *__restrict__ cols, float *__restrict__ vals,
                                                          unsigned long long *__restrict__ nnz) {
    grid_ready();
    __shared__ uint32_t warp_sums[8], off[256], cnt[256];
    __shared__ const uint2 *first[256];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tile = blockIdx.x, capacity = 2 * D.entries;
    const uint32_t hubs = D.words[FZ_HUBS], spare = gridDim.x - tiles;
    const bool apart = hubs <= spare;
    if (tile >= tiles) {
        const uint32_t parts = apart && hubs ? spare / hubs : 1u, b = tile - tiles, h = b / parts;
        if (!apart || h >= hubs) return;
        const uint32_t r = D.longs[h], c = D.count[r], t = r / D.tile_rows;
        if (c <= FZ_WARP_SLOTS) return;  // many partners: written with the others
        uint32_t sum = 0, before;
        for (uint32_t q = t * D.tile_rows + threadIdx.x; q < r; q += 256) sum += D.count[q];
        const uint32_t at = tile_offset(D, t, warp_sums);
        block_scan(sum, warp_sums, before);
        const uint2 *seg = D.hub_out + D.seg[r];
        const uint32_t o = at + before;
        for (uint32_t e = b % parts * 256 + threadIdx.x; e < c && o + e < capacity; e += parts * 256) {
            const uint2 s = seg[e];
            rows[o + e] = r;
            cols[o + e] = s.x;
            vals[o + e] = __uint_as_float(s.y);
        }
        return;
    }
    uint32_t at = tile_offset(D, tile, warp_sums);
    const uint32_t r0 = tile * D.tile_rows, r1 = min(D.n, r0 + D.tile_rows);
    for (uint32_t b = r0; b < r1; b += 256) {
        const uint32_t r = b + threadIdx.x, c = r < r1 ? D.count[r] : 0u;
        first[threadIdx.x] =
            r < r1 ? (D.k + D.indeg[r] > FZ_WARP_SLOTS ? D.hub_out : D.stage) + D.seg[r] : D.stage;
        uint32_t chunk;
        const uint32_t before = block_scan(c, warp_sums, chunk);
        off[threadIdx.x] = at + before;
        cnt[threadIdx.x] = apart && c > FZ_WARP_SLOTS ? 0u : c;
        __syncthreads();
        // two rows a warp, 64 entries of each, loaded before any is stored
        for (uint32_t q = warp; q < min(256u, r1 - b); q += 16) {
            const uint32_t q2 = q + 8;
            const uint32_t c0 = cnt[q], c1 = q2 < 256u ? cnt[q2] : 0u;
            const uint2 *g0 = first[q], *g1 = first[q2 < 256u ? q2 : q];
            for (uint32_t e = lane; e < max(c0, c1); e += 64) {
                uint2 v[4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (e + 32 * h < c0) v[h] = g0[e + 32 * h];
                    if (e + 32 * h < c1) v[2 + h] = g1[e + 32 * h];
                }
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const uint32_t x = e + 32 * (h & 1), row = h < 2 ? q : q2;
                    if (x < (h < 2 ? c0 : c1)) {
                        const uint32_t o = off[row] + x;
                        if (o >= capacity) continue;
                        rows[o] = b + row;
                        cols[o] = v[h].x;
                        vals[o] = __uint_as_float(v[h].y);
                    }
                }
            }
        }
        at += chunk;
        __syncthreads();
    }
    if (tile == tiles - 1 && threadIdx.x == 0) *nnz = at;
}

// Workspace: 36 bytes an entry and about 20 a row, no more than callers sized for when
// the arrivals were sorted.  The hub kernel's output buffer, as large as the segments
// and touched only when there are rows of more than 512 slots, lies over the entries'
// slots, which are used up by then.
struct FuzzyLayout {
    size_t w, slot, stage, hub_out, seg, count, longs, zeroed, zeroed_bytes, bad, total;
    uint32_t tiles, tile_rows;
};

static int fuzzy_layout(uint64_t n, uint32_t k, FuzzyLayout *L) {
    const uint64_t entries = n * k;
    if (n >= 0x7fffffffull || entries > 0x7fffffffull)
        return set_error(HM_ERR_UNSUPPORTED, "n k above 2^31 - 1 entries");
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t here = at;
        at = round_up(at + std::max<size_t>(bytes, 1), 256);
        return here;
    };
    L->tile_rows = (uint32_t)std::max<uint64_t>(FZ_TILE_ROWS, (n + FZ_TILES - 1) / FZ_TILES);
    L->tiles = (uint32_t)((n + L->tile_rows - 1) / L->tile_rows);
    L->w = take(entries * 4);
    L->stage = take(2 * entries * sizeof(uint2));
    L->hub_out = L->slot = take(2 * entries * sizeof(uint2));
    L->seg = take(n * 4);
    L->count = take(n * 4);
    L->longs = take(n * 4);
    // cleared at the start of every run: in-degrees, tile sums, words
    L->zeroed_bytes = (n + L->tiles + FZ_WORDS) * 4;
    L->zeroed = take(L->zeroed_bytes);
    L->bad = L->zeroed + (n + L->tiles + FZ_BAD) * 4;
    L->total = at;
    return HM_OK;
}

}  // namespace hm

using namespace hm;

extern "C" {

size_t hm_fuzzy_workspace_bytes(uint64_t n, uint32_t k) {
    clear_error();
    if (n == 0 || k == 0) {
        set_error(HM_ERR_INVALID, "empty graph");
        return 0;
    }
    FuzzyLayout L;
    if (fuzzy_layout(n, k, &L) != HM_OK) return 0;
    return L.total;
}

int hm_fuzzy_graph_device(const uint32_t *d_idx, const float *d_dist, const float *d_sigma, const float *d_rho,
                          uint64_t n, uint32_t k, uint32_t *d_rows, uint32_t *d_cols, float *d_vals,
                          uint64_t *d_nnz, void *d_workspace, size_t workspace_bytes, void *stream) {
    clear_error();
    if (!d_idx || !d_dist || !d_sigma || !d_rho || !d_rows || !d_cols || !d_vals || !d_nnz || !d_workspace)
        return set_error(HM_ERR_INVALID, "NULL pointer argument");
    if (n == 0 || k == 0) return set_error(HM_ERR_INVALID, "empty graph");
    FuzzyLayout L;
    HM_TRY(fuzzy_layout(n, k, &L));
    if (workspace_bytes < L.total)
        return set_error(HM_ERR_INVALID, "workspace of %zu bytes is below the %zu needed", workspace_bytes, L.total);
    if (reinterpret_cast<uintptr_t>(d_workspace) % 256)
        return set_error(HM_ERR_INVALID, "workspace must be 256-byte aligned");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    char *ws = static_cast<char *>(d_workspace);
    FuzzyDev D{};
    D.idx = d_idx;
    D.dist = d_dist;
    D.sigma = d_sigma;
    D.rho = d_rho;
    D.n = (uint32_t)n;
    D.k = k;
    D.entries = (uint32_t)(n * k);
    D.tile_rows = L.tile_rows;
    D.w = reinterpret_cast<float *>(ws + L.w);
    D.slot = reinterpret_cast<uint32_t *>(ws + L.slot);
    D.stage = reinterpret_cast<uint2 *>(ws + L.stage);
    D.hub_out = reinterpret_cast<uint2 *>(ws + L.hub_out);
    D.seg = reinterpret_cast<uint32_t *>(ws + L.seg);
    D.count = reinterpret_cast<uint32_t *>(ws + L.count);
    D.longs = reinterpret_cast<uint32_t *>(ws + L.longs);
    D.indeg = reinterpret_cast<uint32_t *>(ws + L.zeroed);
    D.tile_sum = D.indeg + n;
    D.words = D.tile_sum + L.tiles;
    const unsigned entry_blocks = (D.entries + 256 * FZ_PER_THREAD - 1) / (256 * FZ_PER_THREAD);
    HM_CUDA_TRY(cudaMemsetAsync(ws + L.zeroed, 0, L.zeroed_bytes, s));
    HM_CUDA_TRY(launch(false, fuzzy_entries_kernel, entry_blocks, 256, 0, s, D));
    HM_CUDA_TRY(launch(true, fuzzy_segments_kernel, (D.n + 255u) / 256u, 256, 0, s, D));
    HM_CUDA_TRY(launch(true, fuzzy_scatter_kernel, entry_blocks, 256, 0, s, D));
    // column and slot share a 32-bit sort key while both fit
    const bool narrow = n < 1ull << (32 - FZ_SLOT_BITS);
    const unsigned union_blocks = (D.n + FZ_WARPS - 1) / FZ_WARPS;
    HM_CUDA_TRY(launch(true, narrow ? fuzzy_union_kernel<uint32_t> : fuzzy_union_kernel<unsigned long long>, union_blocks,
                       FZ_WARPS * 32, 0, s, D));
    // a row's slots: k and, indices not repeating, at most n - 1 sources (the union
    // kernel refuses a longer row where this one does not run)
    if (n + k > FZ_SHORT_SLOTS) {
        auto *kernel = narrow ? fuzzy_long_kernel<uint32_t> : fuzzy_long_kernel<unsigned long long>;
        const size_t bitmaps = (size_t)3 * ((std::min(D.n, FZ_WINDOW) + 31) / 32) * 4, rows_w = 32 * FZ_WARP_SLOTS * 4;
        const size_t part_words = (std::min(D.n, FZ_PART_WINDOW) + 31) / 32, part = part_words * 35 * 4;
        HM_TRY(ensure_dynamic_smem((const void *)kernel, (int)(3 * FZ_WINDOW / 8)));
        HM_CUDA_TRY(launch(true, kernel, device_sm_count(), 1024, std::max({bitmaps, rows_w, part}), s, D));
        count_launch();
    }
    // (a row's entries are distinct columns, repeated indices or not)
    const unsigned spare = n > FZ_WARP_SLOTS ? 4 * device_sm_count() : 0;
    HM_CUDA_TRY(launch(true, fuzzy_write_kernel, L.tiles + spare, 256, 0, s, D, L.tiles, d_rows, d_cols, d_vals,
                       reinterpret_cast<unsigned long long *>(d_nnz)));
    count_launch(5);
    return HM_OK;
}

int hm_fuzzy_graph_status(const void *d_workspace, uint64_t n, uint32_t k, void *stream) {
    clear_error();
    if (!d_workspace) return set_error(HM_ERR_INVALID, "NULL pointer argument");
    FuzzyLayout L;
    HM_TRY(fuzzy_layout(n, k, &L));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    uint32_t bad = 0;
    HM_CUDA_TRY(cudaMemcpyAsync(&bad, static_cast<const char *>(d_workspace) + L.bad, 4,
                                cudaMemcpyDeviceToHost, s));
    HM_CUDA_TRY(cudaStreamSynchronize(s));
    if (bad & FZ_BAD_INDEX) return set_error(HM_ERR_INVALID, "a kNN index is not below n");
    if (bad & FZ_BAD_DUPLICATE) return set_error(HM_ERR_INVALID, "a row of the kNN graph repeats an index");
    return HM_OK;
}

int hm_fuzzy_graph(const uint32_t *idx, const float *dist, const float *sigma, const float *rho, uint64_t n,
                   uint32_t k, uint32_t *rows_out, uint32_t *cols_out, float *vals_out, uint64_t *nnz_out) {
    clear_error();
    if (!idx || !dist || !sigma || !rho || !rows_out || !cols_out || !vals_out || !nnz_out)
        return set_error(HM_ERR_INVALID, "NULL pointer argument");
    if (n == 0 || k == 0) return set_error(HM_ERR_INVALID, "empty graph");
    const uint64_t e = n * k, cap = 2 * e;
    for (uint64_t j = 0; j < e; ++j)
        if (idx[j] >= n) return set_error(HM_ERR_INVALID, "kNN index %u at entry %llu is not below n", idx[j],
                                          (unsigned long long)j);
    for (uint64_t i = 0; i < n; ++i)
        if (sigma[i] < 0.0f) return set_error(HM_ERR_INVALID, "sigma[%llu] is negative", (unsigned long long)i);
    FuzzyLayout L;
    HM_TRY(fuzzy_layout(n, k, &L));
    const size_t ws = L.total;
    // one device block: inputs, outputs, count, workspace (256-byte aligned parts)
    const size_t o_idx = 0, o_dist = round_up(o_idx + e * 4, 256), o_sig = round_up(o_dist + e * 4, 256);
    const size_t o_rho = round_up(o_sig + n * 4, 256), o_rows = round_up(o_rho + n * 4, 256);
    const size_t o_cols = round_up(o_rows + cap * 4, 256), o_vals = round_up(o_cols + cap * 4, 256);
    const size_t o_nnz = round_up(o_vals + cap * 4, 256), o_ws = round_up(o_nnz + 8, 256);
    CallMemory mem;
    HM_TRY(mem.open(o_ws + ws));
    char *const d = mem.p;
    const cudaStream_t s = mem.s;
    int rc = HM_OK;
    uint64_t nnz = 0;
    do {
        cudaError_t err = cudaMemcpyAsync(d + o_idx, idx, e * 4, cudaMemcpyHostToDevice, s);
        if (err == cudaSuccess) err = cudaMemcpyAsync(d + o_dist, dist, e * 4, cudaMemcpyHostToDevice, s);
        if (err == cudaSuccess) err = cudaMemcpyAsync(d + o_sig, sigma, n * 4, cudaMemcpyHostToDevice, s);
        if (err == cudaSuccess) err = cudaMemcpyAsync(d + o_rho, rho, n * 4, cudaMemcpyHostToDevice, s);
        if (err != cudaSuccess) {
            rc = set_error(HM_ERR_CUDA, "copy in: %s", cudaGetErrorString(err));
            break;
        }
        rc = hm_fuzzy_graph_device(reinterpret_cast<uint32_t *>(d + o_idx), reinterpret_cast<float *>(d + o_dist),
                                   reinterpret_cast<float *>(d + o_sig), reinterpret_cast<float *>(d + o_rho), n, k,
                                   reinterpret_cast<uint32_t *>(d + o_rows), reinterpret_cast<uint32_t *>(d + o_cols),
                                   reinterpret_cast<float *>(d + o_vals), reinterpret_cast<uint64_t *>(d + o_nnz),
                                   d + o_ws, ws, s);
        if (rc != HM_OK) break;
        rc = hm_fuzzy_graph_status(d + o_ws, n, k, s);
        if (rc != HM_OK) break;
        err = cudaMemcpyAsync(&nnz, d + o_nnz, 8, cudaMemcpyDeviceToHost, s);
        if (err == cudaSuccess) err = cudaStreamSynchronize(s);
        if (err == cudaSuccess) err = cudaMemcpyAsync(rows_out, d + o_rows, nnz * 4, cudaMemcpyDeviceToHost, s);
        if (err == cudaSuccess) err = cudaMemcpyAsync(cols_out, d + o_cols, nnz * 4, cudaMemcpyDeviceToHost, s);
        if (err == cudaSuccess) err = cudaMemcpyAsync(vals_out, d + o_vals, nnz * 4, cudaMemcpyDeviceToHost, s);
        if (err == cudaSuccess) err = cudaStreamSynchronize(s);
        if (err != cudaSuccess) rc = set_error(HM_ERR_CUDA, "copy out: %s", cudaGetErrorString(err));
    } while (false);
    *nnz_out = nnz;
    return rc;
}

}  // extern "C"
