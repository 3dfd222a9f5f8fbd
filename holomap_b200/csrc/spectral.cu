// spectral.cu -- the normalized graph Laplacian of the fuzzy graph and its
// smallest eigenpairs, the spectral stage that follows the fuzzy graph
// (src/sparse.rs:19-85, src/eigen.rs:31-238, called from spectral_layout_single
// at src/spectral.rs:70-83).
//
// Laplacian (bit-exact with the reference).  From the (row, col)-sorted COO:
//   indptr[r]  = first entry whose row is >= r (src/sparse.rs:21-35 counts rows;
//                on sorted rows both give the same offsets),
//   degree[i]  = sequential binary64 sum of the row's widened weights
//                (src/sparse.rs:57-61),
//   s[p]       = f64(w[p]) * ((1 / sqrt(degree[i])) * (1 / sqrt(degree[j])))
//                (src/sparse.rs:62-69),
// and L x = x - S x with each row's products summed in column order
// (src/sparse.rs:78-84).  Sums start from -0.0, the neutral element of the
// binary64 `Sum` of the reference's toolchain (Rust >= 1.93); it changes
// nothing but the sign of an exactly-zero sum.
//
// Eigenpairs.  Lanczos with locking and warm restarts on B = 2I - L
// following src/eigen.rs:95-223 step for step: the fixed hashed start vector,
// per-cycle Krylov dimension max(8k, 60) (at most n), alpha before the
// re-orthogonalisation, two orthogonalisation passes against the basis and
// the locked vectors, the 1e-12 breakdown test, Ritz pairs of the tridiagonal
// largest first, explicit residual ||B x - theta x|| < 1e-10 to lock, restart
// from the best unconverged Ritz vector, 200 cycles at most, and the
// canonical sign of each vector.  Where the device differs in operation order
// (dot products as fixed two-stage tree reductions; the products L x inside a
// cycle as two chains a lane and a tree per row instead of column order; beta from
// the second orthogonalisation pass's sums; classical Gram-Schmidt, applied twice,
// in place of the modified form; the implicit QL method for the tridiagonal in
// place of nalgebra's SymmetricEigen) the eigenpairs agree with the reference to
// its own tolerances rather than bit for bit.  Every
// reduction has a fixed order, so a graph gives the same bits on every run
// (src/eigen.rs:337-344 asks that of the reference).  The reference uses a
// dense eigensolver when n <= 2000 (src/eigen.rs:31-37); this build runs the
// Lanczos path at every n, as the reference's own spectral parity test does
// for both paths (src/fixture_parity.rs:158-185).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>

#include "hm_internal.cuh"
#include "mbarrier.cuh"

namespace hm {

constexpr unsigned SP_FULL = 0xffffffffu;

// ------------------------------------------------------------- Laplacian

__global__ void csr_indptr_kernel(const uint32_t *__restrict__ rows, uint64_t nnz, uint64_t n,
                                  uint64_t *__restrict__ indptr) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r > n) return;
    uint64_t lo = 0, hi = nnz;
    while (lo < hi) {
        const uint64_t mid = lo + ((hi - lo) >> 1);
        if ((uint64_t)rows[mid] < r) lo = mid + 1;
        else hi = mid;
    }
    indptr[r] = lo;
}

__global__ void degree_kernel(const uint64_t *__restrict__ indptr, const float *__restrict__ vals, uint64_t n,
                              double *__restrict__ deg) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = -0.0;
    for (uint64_t p = indptr[i], e = indptr[i + 1]; p < e; ++p) s = __dadd_rn(s, (double)vals[p]);
    deg[i] = s;
}

__device__ __forceinline__ double inv_sqrt_rn(double d) { return __ddiv_rn(1.0, __dsqrt_rn(d)); }

__global__ void normalize_kernel(const uint32_t *__restrict__ rows, const uint32_t *__restrict__ cols,
                                 const float *__restrict__ vals, uint64_t nnz, const double *__restrict__ deg,
                                 double *__restrict__ svals) {
    const uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nnz) return;
    const double a = inv_sqrt_rn(deg[rows[p]]), b = inv_sqrt_rn(deg[cols[p]]);
    svals[p] = __dmul_rn((double)vals[p], __dmul_rn(a, b));
}

// One warp per row: the products of a 32-entry chunk are formed in parallel,
// then added into the row sum one after another in column order.  Writes y = L x.
__global__ void __launch_bounds__(256) lap_matvec_kernel(const uint64_t *__restrict__ indptr,
                                                         const uint32_t *__restrict__ cols,
                                                         const double *__restrict__ svals, uint64_t n,
                                                         const double *__restrict__ x, double *__restrict__ y) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= n) return;  // whole warps
    const uint64_t lo = indptr[i], hi = indptr[i + 1];
    double acc = -0.0;
    for (uint64_t c0 = lo; c0 < hi; c0 += 32) {
        const uint64_t p = c0 + lane;
        const double prod = p < hi ? __dmul_rn(svals[p], x[cols[p]]) : 0.0;
        const uint32_t cnt = hi - c0 < 32 ? (uint32_t)(hi - c0) : 32u;
        for (uint32_t s = 0; s < cnt; ++s) acc = __dadd_rn(acc, __shfl_sync(SP_FULL, prod, s));
    }
    if (lane == 0) y[i] = __dsub_rn(x[i], acc);
}

// ------------------------------------------------------- Lanczos on the device
// One cooperative launch runs a whole cycle (lanczos_cycle_kernel) and one the
// Ritz vectors of it (ritz_kernel): block b owns the elements [b chunk, (b + 1)
// chunk) of every vector, keeps its part of the basis in shared memory as far
// as it fits (LZ_SMEM_LIMIT), and forms its rows of L x itself, so the blocks meet
// three times a step: after the partial dot products of each orthogonalisation
// pass, and after the new vector is written (the next product gathers all of it).  alpha is the first pass's
// last coefficient, and beta^2 = |w'|^2 - |c2|^2 from the second pass's sums (w'
// after the first pass, c2 its coefficients against the orthonormal basis).
// Dot products are fixed two-stage reductions: every run gives the same bits.
//
// What bounds it: a step of 50,000 points takes about 28 us, 16 of them the
// product's gather from L2 (2.7 M entries; limited by the loads in flight, 26
// bytes a cycle and SM) and 4.5 the three meetings; of 2,000 points 11 us, where
// the phases' fixed costs remain.  Laplacian and 3 eigenpairs, with a launch per
// vector operation and host round trips in every step -> now: 50,000 points
// 22.9 -> 6.7 ms, 12,000 14.7 -> 3.5, 2,000 4.7 -> 1.0; 300,000 48.6 -> 29.2.

constexpr int LZ_THREADS = 1024, LZ_WARPS = LZ_THREADS / 32;
constexpr uint32_t LZ_MAX_BLOCKS = 148;
constexpr uint32_t LZ_MIN_CHUNK = 64;   // elements per block at least: fewer, cheaper meetings
// shared memory of a cycle launch: more would hold more of the basis, but the
// gather's loads in flight live in the L1 that is left (50,000 points: 6.91 ms at
// 176 KB, 6.75 at 144, 6.82 at 80, 7.06 at 16)
constexpr size_t LZ_SMEM_LIMIT = 144 * 1024;
constexpr uint32_t LZ_RITZ = 4;         // Ritz candidates per launch

// the words of LzDev::sync
enum { LZ_ARRIVED = 0, LZ_ERROR = 1, LZ_NSTEPS = 2, LZ_RESTART = 3, LZ_WORDS = 4 };
enum { LZ_START_R = 0, LZ_START_FIRST = 1, LZ_START_SALT = 2 };

// A block's part of the basis: its first `held` rows in shared memory (stride
// `chunk`), the others where all of them are, in global memory (stride n).
struct LzBasis {
    double *sm, *gm;
    uint32_t held;
    uint64_t chunk, n;
    __device__ __forceinline__ double *row(uint32_t u) const { return u < held ? sm + u * chunk : gm + u * n; }
};

struct LzDev {
    const uint64_t *indptr;
    const uint32_t *cols;
    const double *svals;
    uint64_t n;
    uint32_t chunk;         // elements per block
    uint32_t L, steps;      // locked vectors, Krylov dimension of the cycle
    uint32_t held, v_smem;  // basis rows kept in shared memory; the work vector too
    uint32_t start, salt;   // where the cycle's start vector comes from
    double *U;              // locked vectors, then the cycle's basis (rows of n)
    double *w, *r;          // work vector (basis not in shared memory), start vector
    double *part1, *part2;  // block partial sums, [quantity][block]
    double *alpha, *beta;
    uint32_t *sync;
    // Ritz stage
    const double *y;        // per candidate: theta, then its nsteps coefficients
    uint32_t nsteps, take;
    double *X, *resid;      // candidate vectors (rows of n), their residual norms
};

__device__ __forceinline__ double warp_sum_fixed(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(SP_FULL, v, o));
    return v;
}

// All blocks of the cooperative launch meet; false when one did not arrive
// within the limits (every block then leaves, the host reports the error).
__device__ __forceinline__ bool grid_meet(uint32_t *sync, uint32_t &target) {
    __shared__ uint32_t s_ok;
    target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(sync + LZ_ARRIVED) : "memory");
        uint32_t ok = 0;
        const uint64_t t0 = globaltimer_ns();
        for (uint32_t spin = 0; spin < HM_WAIT_SPIN_CAP; ++spin) {
            uint32_t seen;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(sync + LZ_ARRIVED) : "memory");
            if (seen >= target) {
                ok = 1;
                break;
            }
            if ((spin & 255) == 255 && globaltimer_ns() - t0 > HM_WAIT_LIMIT_NS) break;
        }
        if (!ok) atomicExch(&sync[LZ_ERROR], 1u);
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// The block's rows of S as a list of pieces of at most `seg` entries (whole rows,
// or segments of the rows above that: hub rows of a kNN graph hold 20 times the
// average), longest first, so that the warps, taking pieces in turn, finish
// together.  A piece is its first entry (from the block's first) and target |
// length << 12; a target is a row below LZ_LIST_ROWS or LZ_LIST_ROWS + segment.
constexpr uint32_t LZ_LIST_ROWS = 512, LZ_LIST_SEGS = 256, LZ_LIST_MAX = LZ_LIST_ROWS + LZ_LIST_SEGS;
struct LzList {
    uint2 piece[LZ_LIST_MAX + 1];   // one empty piece at the end
    uint32_t seg_of[LZ_LIST_ROWS];  // 0, or first segment << 16 | segments
    double seg_sum[LZ_LIST_SEGS];
    uint64_t first;                 // the block's first entry
    uint32_t count, seg, bucket[5];
};

// Builds the list of rows e0 .. e0 + ne, ne <= LZ_LIST_ROWS (all threads); false
// if their entries do not fit one.
__device__ __forceinline__ bool build_list(const LzDev &D, uint64_t e0, uint64_t ne, LzList &l) {
    if (ne == 0) return false;
    const uint64_t first = D.indptr[e0], entries = D.indptr[e0 + ne] - first;
    // (segments below 256 entries would cost more to combine than they balance)
    const uint64_t seg = max((uint64_t)256, (uint64_t)((entries / (LZ_LIST_SEGS / 2) + 63) & ~63ull));
    if (entries >= 0xffffffffull || seg >= (1u << 20)) return false;
    if (threadIdx.x < 5) l.bucket[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        l.first = first;
        l.seg = (uint32_t)seg;
        l.count = 0;  // segments
    }
    __syncthreads();
    // pieces per bucket of a quarter of seg, then their places: bucket 3 first
    const uint32_t e = threadIdx.x;
    uint32_t lo = 0, len = 0, nseg = 0, seg0 = 0;
    auto bucket_of = [&](uint32_t n) { return n ? min(3u, (uint32_t)((uint64_t)(n - 1) * 4 / seg)) : 0u; };
    if (e < ne) {
        lo = (uint32_t)(D.indptr[e0 + e] - first);
        len = (uint32_t)(D.indptr[e0 + e + 1] - first) - lo;
        nseg = len > seg ? (uint32_t)((len + seg - 1) / seg) : 0u;
        l.seg_of[e] = 0;
        if (nseg) {
            seg0 = atomicAdd(&l.count, nseg);
            l.seg_of[e] = seg0 << 16 | nseg;
            atomicAdd(&l.bucket[3], nseg - 1);
            atomicAdd(&l.bucket[bucket_of(len - (nseg - 1) * (uint32_t)seg)], 1u);
        } else {
            atomicAdd(&l.bucket[bucket_of(len)], 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t at = 0;
        for (int b = 3; b >= 0; --b) {
            const uint32_t c = l.bucket[b];
            l.bucket[b] = at;
            at += c;
        }
        l.count = at;
        l.piece[at] = make_uint2(0u, LZ_LIST_ROWS);
    }
    __syncthreads();
    if (e < ne) {
        for (uint32_t q = 0; q < max(nseg, 1u); ++q) {
            const uint32_t n = nseg ? min((uint32_t)seg, len - q * (uint32_t)seg) : len;
            const uint32_t at = atomicAdd(&l.bucket[bucket_of(n)], 1u);
            l.piece[at] = make_uint2(lo + q * (uint32_t)seg, (nseg ? LZ_LIST_ROWS + seg0 + q : e) | n << 12);
        }
    }
    __syncthreads();
    return true;
}

// Rows e0 .. e0 + ne of S x: a warp on two pieces at a time, 64 entries of each a
// round (a kNN graph's rows hold about 54), the next round's entries loaded while
// this round's gather of x is in flight.  Each lane sums its entries of a piece in
// two chains, then a fixed tree; which warp takes a piece changes nothing.
// f(e, sum) on one thread per row.
template <typename F>
__device__ __forceinline__ void list_matvec(const LzDev &D, const double *x, uint64_t ne, LzList &l, F f) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t *__restrict__ cols = D.cols + l.first + lane;
    const double *__restrict__ svals = D.svals + l.first + lane;
    const uint32_t count = l.count;
    uint32_t at[2], len[2], target[2], c[2][2];
    double v[2][2];
    uint32_t i = 2 * warp, o = 0;
    auto take = [&]() {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint2 p = l.piece[min(i + h, count)];
            at[h] = p.x;
            target[h] = p.y & 4095u;
            len[h] = p.y >> 12;
        }
        o = 0;
    };
    auto load = [&]() {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const bool in = o + 32 * q + lane < len[h];
                c[h][q] = in ? cols[at[h] + o + 32 * q] : 0xffffffffu;
                v[h][q] = in ? svals[at[h] + o + 32 * q] : 0.0;
            }
    };
    take();
    load();
    double a[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    while (i < count) {
        double xv[2][2], vv[2][2];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                xv[h][q] = c[h][q] != 0xffffffffu ? x[c[h][q]] : 0.0;
                vv[h][q] = v[h][q];
            }
        const uint32_t done0 = target[0], done1 = target[1];
        const bool last = o + 64 >= max(len[0], len[1]);
        const uint32_t mine = i;
        o += 64;
        if (last) {
            i += 2 * LZ_WARPS;
            take();
        }
        load();
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 2; ++q) a[h][q] = __fma_rn(vv[h][q], xv[h][q], a[h][q]);
        if (last) {
            double s0 = __dadd_rn(a[0][0], a[0][1]), s1 = __dadd_rn(a[1][0], a[1][1]);
#pragma unroll
            for (int w = 16; w > 0; w >>= 1) {
                s0 = __dadd_rn(s0, __shfl_down_sync(SP_FULL, s0, w));
                s1 = __dadd_rn(s1, __shfl_down_sync(SP_FULL, s1, w));
            }
            if (lane == 0) {
                if (done0 < LZ_LIST_ROWS) f(done0, s0);
                else l.seg_sum[done0 - LZ_LIST_ROWS] = s0;
                if (mine + 1 < count) {
                    if (done1 < LZ_LIST_ROWS) f(done1, s1);
                    else l.seg_sum[done1 - LZ_LIST_ROWS] = s1;
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) a[h][0] = a[h][1] = 0.0;
        }
    }
    __syncthreads();
    if (threadIdx.x < ne && l.seg_of[threadIdx.x]) {
        const uint32_t g0 = l.seg_of[threadIdx.x] >> 16, g1 = g0 + (l.seg_of[threadIdx.x] & 0xffffu);
        double s = 0.0;
        for (uint32_t g = g0; g < g1; ++g) s = __dadd_rn(s, l.seg_sum[g]);
        f(threadIdx.x, s);
    }
}

// The same without a list: a warp per row, 64 entries a round.
template <typename F>
__device__ __forceinline__ void row_matvec(const LzDev &D, const double *x, uint64_t e0, uint64_t ne, F f) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint64_t e = warp; e < ne; e += LZ_WARPS) {
        const uint64_t lo = D.indptr[e0 + e], hi = D.indptr[e0 + e + 1];
        double a = 0.0, b = 0.0;
        for (uint64_t p = lo + lane; p < hi; p += 64) {
            a = __fma_rn(D.svals[p], x[D.cols[p]], a);
            if (p + 32 < hi) b = __fma_rn(D.svals[p + 32], x[D.cols[p + 32]], b);
        }
        const double s = warp_sum_fixed(__dadd_rn(a, b));
        if (lane == 0) f(e, s);
    }
}

// The block's rows of S x: by its list, or, in chunks of several lists' rows, list
// by list (each built again for every product).
template <typename F>
__device__ __forceinline__ void chunk_matvec(const LzDev &D, const double *x, uint64_t e0, uint64_t ne, bool listed,
                                             LzList &l, F f) {
    for (uint64_t t0 = 0; t0 < ne; t0 += LZ_LIST_ROWS) {
        const uint64_t nt = min((uint64_t)LZ_LIST_ROWS, ne - t0);
        auto row = [&](uint64_t e, double s) { f(t0 + e, s); };
        if (ne > LZ_LIST_ROWS) {
            __syncthreads();
            listed = build_list(D, e0 + t0, nt, l);
        }
        if (listed) list_matvec(D, x, nt, l, row);
        else row_matvec(D, x, e0 + t0, nt, row);
    }
    __syncthreads();
}

// This block's part of the dot products of v with the first nu rows of U (and with
// itself, last, if `norm`): part[u * blocks + block].  A group of 8 to 32 lanes
// per product, the widest at which the block takes all products at once; in long
// chunks several warps per product while there are fewer products than warps.
__device__ __forceinline__ void chunk_dots(const LzBasis &U, uint32_t nu, bool norm, const double *v, uint64_t ne,
                                           double *part, double *red) {
    const uint32_t total = nu + (norm ? 1u : 0u);
    if (total == 0) return;
    const uint32_t lg = total <= LZ_WARPS ? 5u : (total <= 2 * LZ_WARPS ? 4u : 3u), lanes = 1u << lg;
    uint32_t lseg = total >= LZ_WARPS ? 0u : (uint32_t)__clz(total - 1) - 27u;
    while (lseg && ((uint64_t)256 << lseg) > ne) --lseg;
    const uint32_t sub = threadIdx.x & (lanes - 1), items = total << lseg;
    const uint64_t hop = (uint64_t)lanes << lseg;
    for (uint32_t it = threadIdx.x >> lg; it < ((items + 3) & ~3u); it += LZ_THREADS >> lg) {  // whole warps
        const uint32_t u = it >> lseg;
        const double *row = u < nu ? U.row(u) : v;
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        uint64_t e = ((uint64_t)(it & ((1u << lseg) - 1)) << lg) + sub;
        for (; e + 3 * hop < ne; e += 4 * hop)
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) s[q] = __fma_rn(row[e + q * hop], v[e + q * hop], s[q]);
        for (; e < ne; e += hop) s[0] = __fma_rn(row[e], v[e], s[0]);
        s[0] = __dadd_rn(__dadd_rn(s[0], s[1]), __dadd_rn(s[2], s[3]));
        for (uint32_t o = lanes >> 1; o > 0; o >>= 1) s[0] = __dadd_rn(s[0], __shfl_down_sync(SP_FULL, s[0], o, lanes));
        if (sub == 0 && it < items) {
            if (lseg) red[it] = s[0];
            else part[(uint64_t)u * gridDim.x + blockIdx.x] = s[0];
        }
    }
    if (lseg) {
        __syncthreads();
        if (threadIdx.x < total) {
            double s = 0.0;
            for (uint32_t g = 0; g < (1u << lseg); ++g) s = __dadd_rn(s, red[(threadIdx.x << lseg) + g]);
            part[(uint64_t)threadIdx.x * gridDim.x + blockIdx.x] = s;
        }
    }
}

// c[u] = the blocks' partial sums of quantity u, u < total (every block forms
// all of them, in the same order), 8 lanes each: up to 128 at once, so the
// whole reduction waits for L2 once
template <uint32_t NV>
__device__ __forceinline__ void reduce_lanes(const double *part, uint32_t total, double *c) {
    const uint32_t sub = threadIdx.x & 7, nb = gridDim.x;
    for (uint32_t u = threadIdx.x >> 3; u < ((total + 3) & ~3u); u += LZ_THREADS / 8) {  // whole warps
        const double *row = part + (uint64_t)min(u, total - 1) * nb;
        double v[NV];
#pragma unroll
        for (uint32_t q = 0; q < NV; ++q) v[q] = sub + 8 * q < nb ? row[sub + 8 * q] : 0.0;
#pragma unroll
        for (uint32_t w = 1; w < NV; w *= 2)  // pairwise
#pragma unroll
            for (uint32_t q = 0; q + w < NV; q += 2 * w) v[q] = __dadd_rn(v[q], v[q + w]);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) v[0] = __dadd_rn(v[0], __shfl_down_sync(SP_FULL, v[0], o, 8));
        if (sub == 0 && u < total) c[u] = v[0];
    }
}
__device__ __forceinline__ void reduce_parts(const double *part, uint32_t total, double *c) {
    if (total && gridDim.x <= 32) reduce_lanes<4>(part, total, c);
    else if (total) reduce_lanes<(LZ_MAX_BLOCKS + 7) / 8>(part, total, c);
    __syncthreads();
}

// How a block's threads share its elements in chunk_project: `parts` threads per
// element while the chunk leaves threads idle (0: one, striding over the chunk).
struct LzSplit {
    uint32_t wide, parts, p, e;
};
__device__ __forceinline__ LzSplit split_of(uint64_t ne) {
    LzSplit s{};
    s.wide = (uint32_t)min((ne + 31) & ~31ull, (unsigned long long)LZ_THREADS);
    s.parts = ne && ne <= LZ_THREADS / 2 ? min(LZ_THREADS / s.wide, 8u) : 0u;
    if (s.parts) {
        s.p = threadIdx.x / s.wide;
        s.e = threadIdx.x - s.p * s.wide;
    }
    return s;
}

// v -= sum over u of c[u] U[u]
__device__ __forceinline__ void chunk_project(const LzBasis &U, uint32_t nu, const double *c,
                                              double *v, uint64_t ne, const LzSplit &sp, double *red) {
    const uint32_t parts = max(sp.parts, 1u);
    auto column = [&](uint64_t e, uint32_t u0) {
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        uint32_t u = u0;
        const uint32_t held = min(U.held, nu);
        const double *at = U.sm + u0 * U.chunk + e;
        for (; u + parts < held; u += 2 * parts, at += 2 * parts * U.chunk) {
            s[0] = __fma_rn(c[u], at[0], s[0]);
            s[1] = __fma_rn(c[u + parts], at[parts * U.chunk], s[1]);
        }
        if (u < held) {
            s[0] = __fma_rn(c[u], at[0], s[0]);
            u += parts;
        }
        at = U.gm + u * U.n + e;
        for (; u < nu; u += 4 * parts, at += 4 * parts * U.n) {
            double x[4];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) x[q] = u + q * parts < nu ? at[q * parts * U.n] : 0.0;
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                if (u + q * parts < nu) s[q] = __fma_rn(c[u + q * parts], x[q], s[q]);
        }
        return __dadd_rn(__dadd_rn(s[0], s[1]), __dadd_rn(s[2], s[3]));
    };
    if (!sp.parts) {
        for (uint64_t e = threadIdx.x; e < ne; e += LZ_THREADS) v[e] = __dsub_rn(v[e], column(e, 0));
    } else {
        if (sp.p < parts && sp.e < ne) red[threadIdx.x] = column(sp.e, sp.p);
        __syncthreads();
        if (threadIdx.x < ne) {
            double s = red[threadIdx.x];
            for (uint32_t q = 1; q < parts; ++q) s = __dadd_rn(s, red[q * sp.wide + threadIdx.x]);
            v[threadIdx.x] = __dsub_rn(v[threadIdx.x], s);
        }
    }
    __syncthreads();
}

// Knuth multiplicative hash in [0, 1) (src/eigen.rs:66-72)
__device__ __forceinline__ double hash01(uint64_t i, uint32_t salt) {
    const uint32_t h = ((uint32_t)i + salt) * 2654435761u;
    return __ddiv_rn((double)(h >> 8), (double)(1u << 24));
}

// One Lanczos cycle (src/eigen.rs:95-168): start vector, its orthogonalisation
// against the locked vectors, then up to `steps` basis vectors.
__global__ void __launch_bounds__(LZ_THREADS, 1) lanczos_cycle_kernel(const LzDev D) {
    extern __shared__ __align__(16) double lz_smem[];
    __shared__ double red[LZ_THREADS];
    __shared__ double s_beta;
    __shared__ LzList list;
    const uint32_t tid = threadIdx.x;
    const uint64_t n = D.n, e0 = min(n, (uint64_t)blockIdx.x * D.chunk), ne = min((uint64_t)D.chunk, n - e0);
    const uint32_t rows = D.L + D.steps;
    double *c = lz_smem;                       // rows + 1 coefficients
    double *usm = c + ((rows + 2) & ~1u);      // held rows of the basis, then the work vector
    double *const v = D.v_smem ? usm + (size_t)D.held * D.chunk : D.w + e0;
    const LzBasis U{usm, D.U + e0, D.held, D.chunk, n};
    uint32_t target = 0;
    const bool listed = ne <= LZ_LIST_ROWS && build_list(D, e0, ne, list);
    const LzSplit split = split_of(ne);

    for (uint64_t e = tid; e < ne; e += LZ_THREADS) {
        const uint64_t i = e0 + e;
        v[e] = D.start == LZ_START_R       ? D.r[i]
               : D.start == LZ_START_FIRST ? __dadd_rn(1.0, __dmul_rn(0.01, __dsub_rn(hash01(i, 0), 0.5)))
                                           : __dsub_rn(hash01(i, D.salt), 0.5);
    }
    for (uint32_t u = 0; u < min(D.L, D.held); ++u)
        for (uint64_t e = tid; e < ne; e += LZ_THREADS) usm[(uint64_t)u * D.chunk + e] = D.U[(uint64_t)u * n + e0 + e];
    __syncthreads();
    // Round j = -1 orthogonalises the start vector against the locked ones,
    // round j >= 0 forms B v_j and orthogonalises it against them and the basis
    // so far; both end with the next basis vector.  (One copy of each phase: the
    // block runs a few hundred instructions of each per step, and refetching
    // several inlined copies cost more than the work.)
    double *basis = D.U + (uint64_t)D.L * n;
    uint32_t nsteps = 0;
    for (int64_t j = -1;; ++j) {
        const uint32_t nu = (uint32_t)(D.L + j + 1);
        if (j >= 0) {
            const double *own = U.row(nu - 1);
            auto row = [&](uint64_t e, double sx) {
                const double xi = own[e];
                v[e] = __dsub_rn(__dmul_rn(2.0, xi), __dsub_rn(xi, sx));
            };
            chunk_matvec(D, basis + (uint64_t)j * n, e0, ne, listed, list, row);
        }
#pragma unroll 1
        for (uint32_t pass = 0; pass < 2; ++pass) {
            double *part = pass ? D.part2 : D.part1;
            chunk_dots(U, nu, pass != 0, v, ne, part, red);
            if (!grid_meet(D.sync, target)) return;
            reduce_parts(part, nu + pass, c);
            if (pass == 0) {
                if (j >= 0 && blockIdx.x == 0 && tid == 0) D.alpha[j] = c[nu - 1];
                if (j >= 0 && ++nsteps == D.steps) break;
            } else if (tid < 32) {
                double s = 0.0;
                for (uint32_t u = tid; u < nu; u += 32) s = __fma_rn(c[u], c[u], s);
                s = warp_sum_fixed(s);
                // (a NaN stays one, so that the tridiagonal solver refuses the graph)
                const double sq = __dsub_rn(c[nu], s);
                if (tid == 0) s_beta = __dsqrt_rn(sq < 0.0 ? 0.0 : sq);
            }
            chunk_project(U, nu, c, v, ne, split, red);  // ends with the block's barrier
        }
        if (nsteps == D.steps) break;
        const double beta = s_beta;
        if (beta < 1e-12) {  // the start vector lies in the locked space, or the basis is invariant
            if (j < 0) {
                if (blockIdx.x == 0 && tid == 0) D.sync[LZ_RESTART] = 1;
                return;
            }
            break;
        }
        if (j >= 0 && blockIdx.x == 0 && tid == 0) D.beta[j] = beta;
        for (uint64_t e = tid; e < ne; e += LZ_THREADS) {
            const double x = __ddiv_rn(v[e], beta);
            basis[(uint64_t)(j + 1) * n + e0 + e] = x;
            if (nu < D.held) usm[(uint64_t)nu * D.chunk + e] = x;
        }
        if (!grid_meet(D.sync, target)) return;
    }
    if (blockIdx.x == 0 && tid == 0) D.sync[LZ_NSTEPS] = nsteps;
}

// Up to LZ_RITZ Ritz vectors x = V y, normalised, and their residual norms
// |2 x - L x - theta x| (src/eigen.rs:180-203).
__global__ void __launch_bounds__(LZ_THREADS, 1) ritz_kernel(const LzDev D) {
    __shared__ double c[LZ_RITZ], red[LZ_WARPS];
    __shared__ LzList list;
    const uint32_t tid = threadIdx.x;
    const uint64_t n = D.n, e0 = min(n, (uint64_t)blockIdx.x * D.chunk), ne = min((uint64_t)D.chunk, n - e0);
    const double *V = D.U + (uint64_t)D.L * n + e0;
    const uint32_t row = D.nsteps + 1;  // doubles per candidate in y
    uint32_t target = 0;
    const bool listed = ne <= LZ_LIST_ROWS && build_list(D, e0, ne, list);
    for (uint64_t e = tid; e < ne; e += LZ_THREADS) {
        double a[LZ_RITZ] = {};
        for (uint32_t s = 0; s < D.nsteps; ++s) {
            const double vs = V[(uint64_t)s * n + e];
#pragma unroll
            for (uint32_t q = 0; q < LZ_RITZ; ++q)
                if (q < D.take) a[q] = __fma_rn(D.y[q * row + 1 + s], vs, a[q]);
        }
#pragma unroll
        for (uint32_t q = 0; q < LZ_RITZ; ++q)
            if (q < D.take) D.X[(uint64_t)q * n + e0 + e] = a[q];
    }
    __syncthreads();
    for (uint32_t q = 0; q < D.take; ++q) {
        chunk_dots(LzBasis{}, 0, true, D.X + (uint64_t)q * n + e0, ne, D.part1 + (uint64_t)q * gridDim.x, red);
        __syncthreads();
    }
    if (!grid_meet(D.sync, target)) return;
    reduce_parts(D.part1, D.take, c);
    for (uint32_t q = 0; q < D.take; ++q) {
        const double norm = __dsqrt_rn(c[q]);
        for (uint64_t e = tid; e < ne; e += LZ_THREADS) {
            double *x = D.X + (uint64_t)q * n + e0 + e;
            *x = __ddiv_rn(*x, norm);
        }
    }
    if (!grid_meet(D.sync, target)) return;
    for (uint32_t q = 0; q < D.take; ++q) {
        const double *x = D.X + (uint64_t)q * n;
        const double theta = D.y[q * row];
        double *z = D.w + e0;
        auto residual = [&](uint64_t e, double sx) {
            const double xi = x[e0 + e], lx = __dsub_rn(xi, sx);
            z[e] = __dsub_rn(__dsub_rn(__dmul_rn(2.0, xi), lx), __dmul_rn(theta, xi));
        };
        chunk_matvec(D, x, e0, ne, listed, list, residual);
        chunk_dots(LzBasis{}, 0, true, z, ne, D.part2 + (uint64_t)q * gridDim.x, red);
        __syncthreads();
    }
    if (!grid_meet(D.sync, target)) return;
    if (blockIdx.x == 0) {
        reduce_parts(D.part2, D.take, c);
        if (tid < D.take) D.resid[tid] = __dsqrt_rn(c[tid]);
    }
}

// ------------------------------------------------------ tridiagonal eigen (host)
// Eigenvalues and eigenvectors of the symmetric tridiagonal matrix with
// diagonal d[0..m) and off-diagonal e[0..m-1): the implicit QL method with
// Wilkinson shifts and plane rotations (Bowdler, Martin, Reinsch and
// Wilkinson, "The QR and QL algorithms for symmetric matrices", 1968; the
// tql2 procedure).  z (m x m) receives eigenvector i as row i, so a rotation
// runs over two contiguous rows.  Returns false if an eigenvalue needs more than
// 60 sweeps.
static inline double pythag(double a, double b) {  // hypot's scaling only where squares underflow
    const double h = a * a + b * b;
    return h > 1e-280 && h < 1e280 ? std::sqrt(h) : std::hypot(a, b);
}
static bool tridiag_eigen(std::vector<double> &d, std::vector<double> e, std::vector<double> &z) {
    const int m = (int)d.size();
    e.resize(m, 0.0);
    e[m - 1] = 0.0;
    z.assign((size_t)m * m, 0.0);
    for (int i = 0; i < m; ++i) z[(size_t)i * m + i] = 1.0;
    for (int l = 0; l < m; ++l) {
        int iter = 0;
        for (;;) {
            int mm = l;
            for (; mm < m - 1; ++mm) {
                const double dd = std::fabs(d[mm]) + std::fabs(d[mm + 1]);
                if (std::fabs(e[mm]) <= DBL_EPSILON * dd) break;
            }
            if (mm == l) break;
            if (++iter > 60) return false;
            double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
            double r = pythag(g, 1.0);
            g = d[mm] - d[l] + e[l] / (g + std::copysign(r, g));
            double s = 1.0, c = 1.0, p = 0.0;
            bool deflated = false;
            for (int i = mm - 1; i >= l; --i) {
                double f = s * e[i];
                const double b = c * e[i];
                r = pythag(f, g);
                e[i + 1] = r;
                if (r == 0.0) {
                    d[i + 1] -= p;
                    e[mm] = 0.0;
                    deflated = true;
                    break;
                }
                s = f / r;
                c = g / r;
                g = d[i + 1] - p;
                r = (d[i] - g) * s + 2.0 * c * b;
                p = s * r;
                d[i + 1] = g + p;
                g = c * r - b;
                double *zi = z.data() + (size_t)i * m, *zn = zi + m;
                for (int q = 0; q < m; ++q) {
                    const double hi = zn[q], lo = zi[q];
                    zn[q] = s * lo + c * hi;
                    zi[q] = c * lo - s * hi;
                }
            }
            if (deflated) continue;
            d[l] -= p;
            e[l] = g;
            e[mm] = 0.0;
        }
    }
    return true;
}

// canonical sign (src/eigen.rs:74-90): the first component of largest
// magnitude (by more than 1e-15) is made positive
static void canonical_sign(double *v, uint64_t n) {
    uint64_t pivot = 0;
    for (uint64_t i = 0; i < n; ++i)
        if (std::fabs(v[i]) > std::fabs(v[pivot]) + 1e-15) pivot = i;
    if (v[pivot] < 0.0)
        for (uint64_t i = 0; i < n; ++i) v[i] = -v[i];
}

// Blocks of the cooperative launches: at least LZ_MIN_CHUNK elements each, at
// most one block per SM.
static uint32_t lz_blocks(uint64_t n) {
    const uint64_t want = (n + LZ_MIN_CHUNK - 1) / LZ_MIN_CHUNK;
    return (uint32_t)std::min<uint64_t>(want, std::min<uint32_t>(LZ_MAX_BLOCKS, (uint32_t)device_sm_count()));
}

// One Lanczos run (src/eigen.rs:95-223): the host drives the cycles, solves the
// tridiagonal and decides what to lock.
struct Lanczos {
    LzDev D{};
    uint32_t k = 0, m = 0, blocks = 0;
    double *stat = nullptr;  // alpha, beta, resid and the sync words, read back in one copy
    uint32_t stat_rows = 0;
    double *ritz = nullptr;  // block partials of the Ritz stage
    cudaStream_t s = nullptr;

    int launch(const void *kernel, size_t smem) {
        HM_CUDA_TRY(cudaMemsetAsync(D.sync, 0, LZ_WORDS * sizeof(uint32_t), s));
        void *args[] = {&D};
        HM_CUDA_TRY(cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(LZ_THREADS), args, smem, s));
        count_launch();
        return HM_OK;
    }
    // alpha, beta, resid and the sync words to the host; the status of the launch
    int read(std::vector<double> &h, uint32_t *words) {
        h.resize((size_t)2 * stat_rows + LZ_RITZ + LZ_WORDS / 2);
        HM_CUDA_TRY(cudaMemcpyAsync(h.data(), stat, h.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        HM_CUDA_TRY(cudaStreamSynchronize(s));
        std::memcpy(words, h.data() + 2 * (size_t)stat_rows + LZ_RITZ, LZ_WORDS * sizeof(uint32_t));
        if (words[LZ_ERROR]) return set_error(HM_ERR_TIMEOUT, "a Lanczos block gave up waiting");
        return HM_OK;
    }

    // values_out / vectors_out (column-major n x found)
    int run(double *values_out, double *vectors_out, uint32_t *found_out, uint32_t *cycles_out) {
        const double LOCK_TOL = 1e-10;
        const uint32_t MAX_CYCLES = 200;
        const uint64_t n = D.n;
        std::vector<double> locked_vals, h, theta, beta_h, z, ybuf;
        uint32_t words[LZ_WORDS];
        uint32_t L = 0, cycle = 0;
        D.start = LZ_START_FIRST;
        while (L < k && cycle < MAX_CYCLES) {
            ++cycle;
            D.L = L;
            D.steps = (uint32_t)std::min<uint64_t>(m, n - L);
            // shared memory: the coefficients, the work vector, and as much of the
            // basis as leaves the product's gather its L1
            const size_t coef = ((size_t)L + D.steps + 2) * sizeof(double), part = (size_t)D.chunk * sizeof(double);
            D.v_smem = coef + part <= LZ_SMEM_LIMIT ? 1u : 0u;
            D.held = D.v_smem ? (uint32_t)std::min<size_t>(L + D.steps, (LZ_SMEM_LIMIT - coef - part) / part) : 0u;
            const size_t smem = coef + (D.v_smem ? (D.held + 1) * part : 0);
            const void *kernel = (const void *)lanczos_cycle_kernel;
            HM_TRY(ensure_dynamic_smem(kernel, (int)std::max(LZ_SMEM_LIMIT, coef)));
            HM_TRY(launch(kernel, smem));
            HM_TRY(read(h, words));
            if (words[LZ_RESTART]) {  // the start vector lies in the locked space
                D.start = LZ_START_SALT;
                D.salt = cycle;
                continue;
            }
            // Ritz pairs of the tridiagonal, largest theta first
            const uint32_t nsteps = D.nsteps = words[LZ_NSTEPS];
            theta.assign(h.begin(), h.begin() + nsteps);
            beta_h.assign(h.begin() + stat_rows, h.begin() + stat_rows + (nsteps - 1));
            if (!tridiag_eigen(theta, beta_h, z))
                return set_error(HM_ERR_UNSUPPORTED, "tridiagonal eigensolver did not converge");
            std::vector<uint32_t> order(nsteps);
            for (uint32_t q = 0; q < nsteps; ++q) order[q] = q;
            std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return theta[a] > theta[b]; });
            const uint32_t take = std::min<uint32_t>(nsteps, k - L + 1);
            std::vector<double> resid(take);
            double *const X0 = D.X, *const part1 = D.part1, *const part2 = D.part2;
            for (uint32_t c0 = 0; c0 < take; c0 += LZ_RITZ) {
                D.take = std::min<uint32_t>(LZ_RITZ, take - c0);
                ybuf.resize((size_t)D.take * (nsteps + 1));
                for (uint32_t c = 0; c < D.take; ++c) {
                    const uint32_t col = order[c0 + c];
                    ybuf[(size_t)c * (nsteps + 1)] = theta[col];
                    for (uint32_t q = 0; q < nsteps; ++q)
                        ybuf[(size_t)c * (nsteps + 1) + 1 + q] = z[(size_t)col * nsteps + q];
                }
                // (into the rows of U past the cycle's basis: see lanczos_layout)
                double *const y = D.U + ((uint64_t)L + nsteps) * n;
                D.y = y;
                HM_CUDA_TRY(cudaMemcpyAsync(y, ybuf.data(), ybuf.size() * sizeof(double), cudaMemcpyHostToDevice, s));
                D.X = X0 + (uint64_t)c0 * n;
                D.part1 = ritz;
                D.part2 = ritz + (size_t)LZ_RITZ * blocks;
                const int rc = launch((const void *)ritz_kernel, 0);
                D.X = X0;
                D.part1 = part1;
                D.part2 = part2;
                if (rc != HM_OK) return rc;
                HM_TRY(read(h, words));
                for (uint32_t c = 0; c < D.take; ++c) resid[c0 + c] = h[2 * (size_t)stat_rows + c];
            }
            // lock converged pairs; warm-restart from the best unconverged one
            bool have_next = false;
            for (uint32_t c = 0; c < take; ++c) {
                const double *xc = D.X + (uint64_t)c * n;
                if (resid[c] < LOCK_TOL && L < k) {
                    HM_CUDA_TRY(cudaMemcpyAsync(D.U + (uint64_t)L * n, xc, n * sizeof(double), cudaMemcpyDeviceToDevice,
                                                s));
                    locked_vals.push_back(2.0 - theta[order[c]]);
                    ++L;
                } else if (!have_next) {
                    HM_CUDA_TRY(cudaMemcpyAsync(D.r, xc, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
                    have_next = true;
                }
            }
            D.start = have_next ? LZ_START_R : LZ_START_SALT;
            D.salt = cycle;
        }
        // ascending lambda, canonical orientation
        std::vector<uint32_t> idx(L);
        for (uint32_t q = 0; q < L; ++q) idx[q] = q;
        std::stable_sort(idx.begin(), idx.end(), [&](uint32_t a, uint32_t b) { return locked_vals[a] < locked_vals[b]; });
        const uint32_t found = std::min(k, L);
        for (uint32_t j = 0; j < found; ++j) {
            values_out[j] = locked_vals[idx[j]];
            double *out = vectors_out + (uint64_t)j * n;
            HM_CUDA_TRY(cudaMemcpyAsync(out, D.U + (uint64_t)idx[j] * n, n * sizeof(double), cudaMemcpyDeviceToHost, s));
        }
        HM_CUDA_TRY(cudaStreamSynchronize(s));
        for (uint32_t j = 0; j < found; ++j) canonical_sign(vectors_out + (uint64_t)j * n, n);
        *found_out = found;
        if (cycles_out) *cycles_out = cycle;
        return HM_OK;
    }
};

static int laplacian_launch(const uint32_t *d_rows, const uint32_t *d_cols, const float *d_vals, uint64_t n,
                            uint64_t nnz, uint64_t *d_indptr, double *d_svals, double *d_degrees, cudaStream_t s) {
    csr_indptr_kernel<<<(unsigned)((n + 1 + 255) / 256), 256, 0, s>>>(d_rows, nnz, n, d_indptr);
    HM_CUDA_TRY(cudaGetLastError());
    degree_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_indptr, d_vals, n, d_degrees);
    HM_CUDA_TRY(cudaGetLastError());
    count_launch(2);
    if (nnz) {
        normalize_kernel<<<(unsigned)((nnz + 255) / 256), 256, 0, s>>>(d_rows, d_cols, d_vals, nnz, d_degrees,
                                                                      d_svals);
        HM_CUDA_TRY(cudaGetLastError());
        count_launch();
    }
    return HM_OK;
}

// Workspace of an eigenpair run (beyond the Laplacian itself), in bytes from its
// start; no larger than callers sized for when every step was its own launches.  The
// block partials of a cycle lie in the candidates' room (the two are never live
// together).  The candidates' coefficients lie in the rows of U past the cycle's
// basis: a cycle with L locked vectors has at most k + 1 - L candidates of nsteps + 1
// <= n + 1 coefficients each, and at least k + 1 - L rows are free.
struct LzLayout {
    size_t U, X, w, r, ritz, stat, total;
    uint32_t m, rows, blocks;
};
static LzLayout lanczos_layout(uint64_t n, uint32_t k) {
    LzLayout l{};
    l.m = (uint32_t)std::min<uint64_t>(n, std::max<uint32_t>(8 * k, 60));
    l.rows = k + l.m + 1;
    l.blocks = (uint32_t)std::min<uint64_t>((n + LZ_MIN_CHUNK - 1) / LZ_MIN_CHUNK, LZ_MAX_BLOCKS);
    size_t at = 0;
    auto take = [&](size_t doubles) {
        const size_t here = at;
        at += round_up(doubles * sizeof(double), 256);
        return here;
    };
    l.U = take((size_t)l.rows * n + LZ_RITZ);
    l.X = take(std::max<size_t>((size_t)(k + 1) * n, (size_t)2 * (l.rows + 1) * l.blocks));
    l.w = take(n);
    l.r = take(n);
    l.ritz = take((size_t)2 * LZ_RITZ * l.blocks);
    l.stat = take((size_t)2 * l.rows + LZ_RITZ + LZ_WORDS / 2);
    l.total = at;
    return l;
}

}  // namespace hm

using namespace hm;

extern "C" {

int hm_laplacian_device(const uint32_t *d_rows, const uint32_t *d_cols, const float *d_vals, uint64_t n,
                        uint64_t nnz, uint64_t *d_indptr, double *d_svals, double *d_degrees, void *stream) {
    clear_error();
    if (!d_rows || !d_cols || !d_vals || !d_indptr || !d_svals || !d_degrees)
        return set_error(HM_ERR_INVALID, "NULL pointer argument");
    if (n == 0) return set_error(HM_ERR_INVALID, "empty graph");
    return laplacian_launch(d_rows, d_cols, d_vals, n, nnz, d_indptr, d_svals, d_degrees,
                            static_cast<cudaStream_t>(stream));
}

int hm_laplacian_matvec_device(const uint64_t *d_indptr, const uint32_t *d_cols, const double *d_svals,
                               uint64_t n, const double *d_x, double *d_y, void *stream) {
    clear_error();
    if (!d_indptr || !d_cols || !d_svals || !d_x || !d_y) return set_error(HM_ERR_INVALID, "NULL pointer argument");
    if (n == 0) return set_error(HM_ERR_INVALID, "empty graph");
    const unsigned blocks = (unsigned)((n * 32 + 255) / 256);
    lap_matvec_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(d_indptr, d_cols, d_svals, n, d_x, d_y);
    HM_CUDA_TRY(cudaGetLastError());
    count_launch();
    return HM_OK;
}

size_t hm_eigenpairs_workspace_bytes(uint64_t n, uint32_t k) {
    clear_error();
    if (n == 0 || k == 0 || k > n) {
        set_error(HM_ERR_INVALID, "need 1 <= k <= n");
        return 0;
    }
    if (k > 1024) {
        set_error(HM_ERR_UNSUPPORTED, "k above 1024");
        return 0;
    }
    return lanczos_layout(n, k).total;
}

int hm_eigenpairs_device(const uint64_t *d_indptr, const uint32_t *d_cols, const double *d_svals, uint64_t n,
                         uint32_t k, void *d_workspace, size_t workspace_bytes, void *stream, double *values_out,
                         double *vectors_out, uint32_t *found_out, uint32_t *cycles_out) {
    clear_error();
    if (!d_indptr || !d_cols || !d_svals || !d_workspace || !values_out || !vectors_out || !found_out)
        return set_error(HM_ERR_INVALID, "NULL pointer argument");
    if (n == 0 || k == 0 || k > n) return set_error(HM_ERR_INVALID, "need 1 <= k <= n");
    if (k > 1024) return set_error(HM_ERR_UNSUPPORTED, "k above 1024");
    if (n > 0xffffffffull) return set_error(HM_ERR_UNSUPPORTED, "n above 2^32 - 1");
    const LzLayout l = lanczos_layout(n, k);
    if (workspace_bytes < l.total)
        return set_error(HM_ERR_INVALID, "workspace of %zu bytes is below the %zu needed", workspace_bytes, l.total);
    if (reinterpret_cast<uintptr_t>(d_workspace) % 256) return set_error(HM_ERR_INVALID, "workspace must be 256-byte aligned");
    auto at = [&](size_t o) { return reinterpret_cast<double *>(static_cast<char *>(d_workspace) + o); };
    Lanczos lz;
    lz.k = k;
    lz.m = l.m;
    lz.blocks = lz_blocks(n);
    lz.s = static_cast<cudaStream_t>(stream);
    lz.stat = at(l.stat);
    lz.stat_rows = l.rows;
    LzDev &D = lz.D;
    D.indptr = d_indptr;
    D.cols = d_cols;
    D.svals = d_svals;
    D.n = n;
    D.chunk = (uint32_t)((n + lz.blocks - 1) / lz.blocks);
    D.U = at(l.U);
    D.X = at(l.X);
    D.w = at(l.w);
    D.r = at(l.r);
    D.part1 = D.X;
    D.part2 = D.X + (size_t)(l.rows + 1) * lz.blocks;
    D.alpha = lz.stat;
    D.beta = lz.stat + l.rows;
    D.resid = lz.stat + 2 * (size_t)l.rows;
    D.sync = reinterpret_cast<uint32_t *>(D.resid + LZ_RITZ);
    lz.ritz = at(l.ritz);
    return lz.run(values_out, vectors_out, found_out, cycles_out);
}

int hm_spectral_eigenpairs(const uint32_t *rows, const uint32_t *cols, const float *vals, uint64_t n, uint64_t nnz,
                           uint32_t k, double *values_out, double *vectors_out, uint32_t *found_out,
                           uint32_t *cycles_out) {
    clear_error();
    if (!rows || !cols || !vals || !values_out || !vectors_out || !found_out)
        return set_error(HM_ERR_INVALID, "NULL pointer argument");
    if (n == 0 || k == 0 || k > n) return set_error(HM_ERR_INVALID, "need 1 <= k <= n");
    for (uint64_t p = 0; p < nnz; ++p) {
        if (rows[p] >= n || cols[p] >= n)
            return set_error(HM_ERR_INVALID, "entry %llu is outside the n x n graph", (unsigned long long)p);
        if (p && rows[p] < rows[p - 1])
            return set_error(HM_ERR_INVALID, "rows are not sorted at entry %llu", (unsigned long long)p);
    }
    const size_t ws = hm_eigenpairs_workspace_bytes(n, k);
    if (ws == 0) return HM_ERR_UNSUPPORTED;
    const size_t o_rows = 0, o_cols = round_up(nnz * 4 + 1, 256), o_vals = o_cols + round_up(nnz * 4 + 1, 256);
    const size_t o_ind = o_vals + round_up(nnz * 4 + 1, 256), o_sv = o_ind + round_up((n + 1) * 8, 256);
    const size_t o_deg = o_sv + round_up(nnz * 8 + 1, 256), o_ws = o_deg + round_up(n * 8, 256);
    CallMemory mem;
    HM_TRY(mem.open(o_ws + ws));
    char *const d = mem.p;
    const cudaStream_t s = mem.s;
    int rc = HM_OK;
    do {
        cudaError_t err = cudaMemcpyAsync(d + o_rows, rows, nnz * 4, cudaMemcpyHostToDevice, s);
        if (err == cudaSuccess) err = cudaMemcpyAsync(d + o_cols, cols, nnz * 4, cudaMemcpyHostToDevice, s);
        if (err == cudaSuccess) err = cudaMemcpyAsync(d + o_vals, vals, nnz * 4, cudaMemcpyHostToDevice, s);
        if (err != cudaSuccess) {
            rc = set_error(HM_ERR_CUDA, "copy in: %s", cudaGetErrorString(err));
            break;
        }
        auto *ind = reinterpret_cast<uint64_t *>(d + o_ind);
        auto *sv = reinterpret_cast<double *>(d + o_sv);
        rc = laplacian_launch(reinterpret_cast<uint32_t *>(d + o_rows), reinterpret_cast<uint32_t *>(d + o_cols),
                              reinterpret_cast<float *>(d + o_vals), n, nnz, ind, sv,
                              reinterpret_cast<double *>(d + o_deg), s);
        if (rc != HM_OK) break;
        rc = hm_eigenpairs_device(ind, reinterpret_cast<uint32_t *>(d + o_cols), sv, n, k, d + o_ws, ws, s,
                                  values_out, vectors_out, found_out, cycles_out);
    } while (false);
    return rc;
}

int hm_debug_tridiag_eigen(const double *d, const double *e, uint32_t m, double *vals_out, double *vecs_out) {
    clear_error();
    if (!d || !vals_out || !vecs_out || (m > 1 && !e) || m == 0) return set_error(HM_ERR_INVALID, "bad arguments");
    std::vector<double> dd(d, d + m), ee(e ? e : d, e ? e + (m - 1) : d), z;
    if (!tridiag_eigen(dd, ee, z)) return set_error(HM_ERR_UNSUPPORTED, "tridiagonal eigensolver did not converge");
    std::memcpy(vals_out, dd.data(), m * sizeof(double));
    for (uint32_t q = 0; q < m; ++q)
        for (uint32_t i = 0; i < m; ++i) vecs_out[(size_t)q * m + i] = z[(size_t)i * m + q];
    return HM_OK;
}

}  // extern "C"
