// plain_knn.cu -- exact kNN over every pair, in the reference's own binary64
// arithmetic, with a warp-level select on (distance bits, index) keys.
//
// Reference: src/knn.rs:22-55 (row loop, self override :35-43, sort by
// (total_cmp(dist), index) and take k :46-52), src/metric.rs:42-53 (euclidean),
// src/metric.rs:58-70 (cosine).
//
// Each pair's distance is the same sequence of correctly rounded binary64
// operations the reference performs: per dimension f64(x) - f64(y), square,
// add to a running sum that starts at +0.0, in dimension order (euclidean), or
// dot += f64(x) * f64(y) (cosine, whose per-row norm sums are precomputed in
// the same order by check_norms_kernel), then sqrt / divide / cast.  A stage's last
// dimensions past d are loaded as zeros and left out of the loop.
//
// Layout: a CTA owns 32 query rows of one job (4 warps x 8 rows) and walks the
// columns of its split 128 at a time; every lane computes an 8x4 block of pairs
// (rows of its warp x columns lane + 32c) from binary64 stages in shared memory,
// widened once per CTA from the binary32 points.  A pair whose accumulator cannot
// reach the row's k-th distance is dropped before its square root or quotient;
// the others are collected 32 at a time and merged into the row's sorted list
// (WarpTopK::merge32), which lives in shared memory.  Column splits write partial
// lists that merge_splits combines.
//
// What bounds it: the binary64 pipe (3 operations per pair and dimension for
// euclidean, 2 manhattan, 1 cosine: the product of two widened binary32 values is
// exact, so the reference's multiply and add are one fused operation).
// Whole calls, with every key inserted one at a time and a separate binary64 copy
// of the points -> now: 1,000 x 50, k = 15 89 -> 58 us; 12,007 x 64 manhattan 1,744
// -> 1,596 us (0.65 of the binary64 rate); 10,000 x 32, k = 100 4,080 -> 1,672 us.
// Registers limit it to 12 warps an SM; 16 (128 registers, spills) measured 2,489
// us on the manhattan call, an unroll of 8 or 16 dimensions 1,668 and 1,875.
#include <cuda_runtime.h>

#include "hm_internal.cuh"

namespace hm {

int kpl_for_k(uint32_t k) {
    if (k <= 32) return 1;
    if (k <= 64) return 2;
    if (k <= 128) return 4;
    if (k <= 256) return 8;
    return 0;
}

// ----------------------------------------------------------------- check
__global__ void init_counters_kernel(JobDev *jobs, uint32_t njobs) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= njobs) return;
    JobCounters c{};
    c.nonfinite_min = 0xffffffffu;
    *jobs[j].cnt = c;
}

// Input check and cosine row norms, one warp per 32 consecutive rows of the
// all-rows space (rows of several jobs may share a warp).  The warp stages its
// rows 32 dimensions at a time through shared memory with coalesced 128-byte
// reads (one row per load instruction), and lane r then walks row r's chunk in
// dimension order: the sequential binary64 sum of squares of the cosine
// metric's na / nb (src/metric.rs:61-66, :69), whose square root is kept per
// row.  Every value read is also checked for finiteness (the smallest flat
// index of a non-finite value per job, as HolomapError::NonFiniteInput
// reports it, src/api.rs:36-43).
constexpr int NRM_WARPS = 8;
__global__ void __launch_bounds__(NRM_WARPS * 32) check_norms_kernel(const JobDev *__restrict__ jobs,
                                                                    uint32_t njobs,
                                                                    const uint32_t *__restrict__ row_starts,
                                                                    uint32_t rows) {
    __shared__ float tile[NRM_WARPS][32][33];
    grid_ready();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t ar0 = (blockIdx.x * NRM_WARPS + warp) * 32;
    if (ar0 >= rows) return;
    const uint32_t ar = ar0 + lane;
    const uint32_t jb = ar < rows ? (row_starts ? find_job(row_starts, njobs, ar) : 0u) : 0u;
    const JobDev &J = jobs[jb];
    // (an escalation copy's rows are its original's: checked there)
    const bool mine = ar < rows && job_active(J);
    const uint32_t row = mine ? ar - J.arow0 : 0u;
    const uint32_t d = mine ? J.d : 0u;
    const float *xrow = J.x + (size_t)row * d;
    const bool cos = mine && J.metric == HM_METRIC_COSINE;
    const uint32_t dmax = __reduce_max_sync(0xffffffffu, d);
    double acc = 0.0;
    for (uint32_t c0 = 0; c0 < dmax; c0 += 32) {
        // row i of the warp, dimension c0 + lane: coalesced per row; all 32
        // rows' loads are issued before any is used
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const float *src = reinterpret_cast<const float *>(
                __shfl_sync(0xffffffffu, reinterpret_cast<uintptr_t>(xrow), i));
            const uint32_t di = __shfl_sync(0xffffffffu, d, i);
            v[i] = (c0 + lane < di) ? src[c0 + lane] : 0.0f;
        }
        uint32_t bad = 0;
#pragma unroll
        for (int i = 0; i < 32; ++i) bad |= isfinite(v[i]) ? 0u : (1u << i);
        bad = __reduce_or_sync(0xffffffffu, bad);
        while (bad) {  // rare: a non-finite value in one of the rows
            const int i = __ffs(bad) - 1;
            bad &= bad - 1;
            const uint32_t di = __shfl_sync(0xffffffffu, d, i);
            const uint32_t ri = __shfl_sync(0xffffffffu, row, i);
            const uint32_t ji = __shfl_sync(0xffffffffu, jb, i);
            float vi = 0.0f;
#pragma unroll
            for (int q = 0; q < 32; ++q) vi = (q == i) ? v[q] : vi;
            if (c0 + lane < di && !isfinite(vi))
                atomicMin(&jobs[ji].cnt->nonfinite_min,
                          (uint32_t)min((size_t)ri * di + c0 + lane, (size_t)0xfffffffeull));
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) tile[warp][i][lane] = v[i];
        __syncwarp();
        if (cos) {
            const uint32_t tmax = min(32u, d - min(d, c0));
            for (uint32_t t = 0; t < tmax; ++t) {
                const double e = (double)tile[warp][lane][t];
                acc = __fma_rn(e, e, acc);  // e * e is exact
            }
        }
        __syncwarp();
    }
    if (cos) J.rnorm[row] = __dsqrt_rn(acc);
}

int launch_check(const JobDev *jobs, uint32_t njobs, const uint32_t *row_starts, uint32_t all_rows, cudaStream_t s) {
    ScopedKernelTimer timer(HM_KCLASS_PREP, s);
    init_counters_kernel<<<(njobs + 127) / 128, 128, 0, s>>>(const_cast<JobDev *>(jobs), njobs);
    HM_CUDA_TRY(cudaGetLastError());
    const uint32_t warps = (all_rows + 31) / 32;
    HM_CUDA_TRY(launch(true, check_norms_kernel, (warps + NRM_WARPS - 1) / NRM_WARPS, NRM_WARPS * 32, 0, s, jobs, njobs,
                       row_starts, all_rows));
    count_launch(2);
    return HM_OK;
}

// ------------------------------------------------------------ the kernel
template <int METRIC>
__device__ __forceinline__ double pair_step(double acc, double a, double b) {
    if (METRIC == HM_METRIC_EUCLIDEAN) {
        const double t = __dsub_rn(a, b);
        return __dadd_rn(acc, __dmul_rn(t, t));
    } else if (METRIC == HM_METRIC_COSINE) {
        return __fma_rn(a, b, acc);  // a * b is exact
    } else {
        return __dadd_rn(acc, fabs(__dsub_rn(a, b)));
    }
}

// Final binary64 -> binary32 step of each metric.
template <int METRIC>
__device__ __forceinline__ float pair_finish(double acc, double rn_a, double rn_b) {
    if (METRIC == HM_METRIC_EUCLIDEAN) {
        return __double2float_rn(__dsqrt_rn(acc));
    } else if (METRIC == HM_METRIC_COSINE) {
        // (1 - dot / (sqrt(na) * sqrt(nb))).max(0.0) as f32; NaN (a zero
        // vector) and any value <= 0 give +0.0.
        const double den = __dmul_rn(rn_a, rn_b);
        const double q = __ddiv_rn(acc, den);
        const double r = __dsub_rn(1.0, q);
        return (r > 0.0) ? __double2float_rn(r) : 0.0f;
    } else {
        return __double2float_rn(acc);
    }
}

// What a pair's accumulator has to reach for its returned distance to be at most
// `dist`, with room for every rounding on the way: one of at most dist comes from a
// value of at most up = dist (1 + 2^-21) + 1.5 * 2^-149.  Euclidean: acc <= up^2 (1 +
// 2^-50); manhattan: acc <= up; cosine: acc >= (1 - up - 2^-44) |a| |b|, returned with
// |a| multiplied in (test it times |b|).
template <int METRIC>
__device__ __forceinline__ double limit_of(double up, double rn_a) {
    if (METRIC == HM_METRIC_EUCLIDEAN) return up * up * (1.0 + 0x1p-50);
    if (METRIC == HM_METRIC_COSINE) {
        const double v = 1.0 - up - 0x1p-44;
        return (v < -1e30 ? -1e30 : v) * rn_a;  // (a NaN stays one)
    }
    return up;
}
template <int METRIC>
__device__ __forceinline__ double pair_limit(float dist, double rn_a) {
    return limit_of<METRIC>((double)dist * (1.0 + 0x1p-21) + 1.5 * 0x1p-149, rn_a);
}
// The limit of a row whose k-th key is tau_key.  The columns come in ascending order,
// so a later pair at exactly the k-th distance tau stays behind it and only a smaller
// distance counts: a value of at most tau (1 - 2^-25), which no midpoint between tau and
// the next smaller binary32 exceeds.  Ties are common where points repeat: at distance
// 0, as all pairs of a zero vector are under cosine, every later pair would be merged for
// nothing (6,000 x 24, k = 15, 300 zero vectors: 1,755 us with ties let through, 1,310
// without).  A row that nothing can enter any more (tau 0) has the limit NaN, which no
// pair reaches; one with fewer than k keys, or an infinite tau, takes every pair.
template <int METRIC>
__device__ __forceinline__ double next_limit(uint64_t tau_key, double rn_a) {
    const float f = __uint_as_float(min((uint32_t)(tau_key >> 32), 0x7f800000u));  // (KEY_NONE: infinity)
    const double tau = (double)(f > 0.0f ? f : __uint_as_float(0x7fffffffu));
    constexpr double below = (1.0 - 0x1p-25) * (1.0 + 0x1p-49);
    if (METRIC == HM_METRIC_EUCLIDEAN) return tau * tau * (below * below);  // (tau * tau is exact)
    return limit_of<METRIC>(tau * below, rn_a);
}

// Shared memory of one CTA.
template <int KPL>
struct PlainSmem {
    double As[2][PL_BM][PL_BK + 1];
    double Bs[2][PL_BN][PL_BK + 1];
    uint64_t list[PL_BM][32 * KPL];  // each row's sorted keys
    uint64_t fresh[PL_BM][64];       // keys waiting to be merged
    double rn_a[PL_BM];
    uint32_t rows[PL_BM];            // the query rows (0xffffffff: none)
    uint32_t last;                   // fallback parts: this one finished last
};

// Merges the first `have` (at most 32) waiting keys into the row's list; returns
// the row's new limit.
template <int METRIC, int KPL>
__device__ __noinline__ double plain_merge(uint64_t *list, const uint64_t *fresh, uint32_t have, uint32_t k,
                                           double rn_a) {
    const int lane = threadIdx.x & 31;
    WarpTopK<KPL> top;
#pragma unroll
    for (int q = 0; q < KPL; ++q) top.v[q] = list[q * 32 + lane];
    const uint64_t b = (uint32_t)lane < have ? fresh[lane] : KEY_NONE;
    top.merge32(b, k, lane);
#pragma unroll
    for (int q = 0; q < KPL; ++q) list[q * 32 + lane] = top.v[q];
    __syncwarp();
    return next_limit<METRIC>(top.tau, rn_a);
}

// The part of a fallback group that finishes last merges the group's lists (its
// counter: see select_row).
template <int KPL>
__device__ __noinline__ void merge_parts(const JobDev &J, PlainSmem<KPL> &sm, uint32_t grp, uint32_t parts) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t k = J.k;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) sm.last = atomicAdd(&J.zero_rows[grp], 1u) == parts - 1 ? 1u : 0u;
    __syncthreads();
    if (!sm.last) return;
    __threadfence();
#pragma unroll 1
    for (int r = 0; r < 8; ++r) {
        const uint32_t row = sm.rows[warp * 8 + r];
        if (row == 0xffffffffu) continue;
        const uint64_t *lists = J.partial + (size_t)row * J.elists * J.cap;
        WarpTopK<KPL> top;
        top.reset();
        for (uint32_t p = 0; p < parts; ++p)
            for (uint32_t e0 = 0; e0 < k; e0 += 32) {
                uint64_t key = KEY_NONE;
                if (e0 + lane < k) key = __ldcg(reinterpret_cast<const unsigned long long *>(lists) + p * k + e0 + lane);
                if (!__any_sync(0xffffffffu, key < top.tau)) break;  // lists are sorted
                top.template merge32<true>(key, k, lane);
            }
#pragma unroll
        for (int q = 0; q < KPL; ++q) {
            const uint32_t e = q * 32 + lane;
            if (e < k) {
                J.idx[(size_t)row * k + e] = key_idx(top.v[q]);
                J.dist[(size_t)row * k + e] = key_dist(top.v[q]);
            }
        }
    }
}

// FALLBACK: the rows are the jobs' overflow lists (a kernel of its own: with both forms
// in one a 700 x 100 call took 68 us, 58 without the fallback's parts).
template <int METRIC, int KPL, bool FALLBACK>
__global__ void __launch_bounds__(PL_THREADS, KPL <= 2 ? 3 : 2) plain_knn_kernel(const PlainWork w) {
    extern __shared__ __align__(16) unsigned char pl_smem_raw[];
    PlainSmem<KPL> &sm = *reinterpret_cast<PlainSmem<KPL> *>(pl_smem_raw);
    grid_ready();
    if (FALLBACK && w.ovf && blockIdx.x >= (*w.ovf + PL_BM - 1) / PL_BM * FB_MAX_PARTS) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint32_t jb, first_grp, grp_stride, n_groups, split = 0, parts = 1;
    if (!FALLBACK) {
        uint32_t lo = 0, hi = w.njobs_m;  // the job whose items hold this block's
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (w.items[mid].y <= blockIdx.x) lo = mid; else hi = mid;
        }
        jb = w.items[lo].x;
        const uint32_t it = blockIdx.x - w.items[lo].y;
        first_grp = w.jobs[jb].q0 / PL_BM + it / w.jobs[jb].splits;
        split = it % w.jobs[jb].splits;
        grp_stride = 1;
        n_groups = first_grp + 1;
    } else {
        jb = w.fb_jobs[blockIdx.x / w.per_job];
        first_grp = blockIdx.x % w.per_job;
        grp_stride = w.per_job;
        n_groups = (w.jobs[jb].cnt->ovf_count + PL_BM - 1) / PL_BM;
        if (first_grp >= n_groups * FB_MAX_PARTS) return;
    }
    const JobDev &J = w.jobs[jb];
    uint32_t split_cols = J.split_cols;
    if (FALLBACK && 2 * n_groups <= w.per_job) {
        // fewer row groups than CTAs: several to a group, a part of the columns each,
        // as many as the row's candidate lists (read for the last time by now) hold lists
        const uint32_t tiles = (J.n + PL_BN - 1) / PL_BN;
        parts = min(min(w.per_job / n_groups, FB_MAX_PARTS), min(tiles, J.elists * J.cap / J.k));
        const uint32_t per = (tiles + parts - 1) / parts;
        parts = (tiles + per - 1) / per;
        split_cols = per * PL_BN;
        split = first_grp % parts;
        first_grp /= parts;
        if (first_grp >= n_groups) return;
        n_groups = first_grp + 1;
    }
    // (a loop the compiler knows to run once costs registers: addresses are hoisted out of
    // it, and the accumulators spill)
    asm volatile("" : "+r"(n_groups));
    const uint32_t c_begin = split * split_cols, c_end = min(J.n, c_begin + split_cols);
    const uint32_t n = J.n, d = J.d, k = J.k;
    const float *__restrict__ x = J.x;
    const bool vec = (d & 3u) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    const uint32_t nk = (d + PL_BK - 1) / PL_BK, tiles = (c_end - c_begin + PL_BN - 1) / PL_BN, stages = tiles * nk;

    for (uint32_t grp = first_grp; grp < n_groups; grp += grp_stride) {
        if (tid < PL_BM) {
            uint32_t r;
            if (FALLBACK) {
                const uint32_t at = grp * PL_BM + tid;
                r = at < J.cnt->ovf_count ? J.ovf_list[at] : 0xffffffffu;
            } else {
                r = grp * PL_BM + tid;
                if (r < J.q0 || r >= J.q1) r = 0xffffffffu;
            }
            sm.rows[tid] = r;
            sm.rn_a[tid] = METRIC == HM_METRIC_COSINE && r != 0xffffffffu ? J.rnorm[r] : 0.0;
        }
        for (uint32_t e = tid; e < PL_BM * 32 * KPL; e += PL_THREADS) sm.list[e / (32 * KPL)][e % (32 * KPL)] = KEY_NONE;
        __syncthreads();

        // A stage: 16 dimensions of the 32 rows and of 128 columns, four values a
        // thread and row: thread t takes row t / 4 (of each 32), dimensions 4 (t % 4)
        const uint32_t lr = tid >> 2, lc = 4 * (tid & 3);
        const uint32_t a_row = min(sm.rows[lr], n - 1);  // no row: any valid one
        float4 nxt[5];
        auto load = [&](uint32_t row, uint32_t dim) {
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (row < n) {
                const float *src = x + (size_t)row * d + dim;
                if (vec && dim < d) {
                    v = *reinterpret_cast<const float4 *>(src);
                } else {
                    if (dim < d) v.x = src[0];
                    if (dim + 1 < d) v.y = src[1];
                    if (dim + 2 < d) v.z = src[2];
                    if (dim + 3 < d) v.w = src[3];
                }
            }
            return v;
        };
        auto fetch = [&](uint32_t col0, uint32_t kt) {
            nxt[0] = load(a_row, kt * PL_BK + lc);
#pragma unroll
            for (int p = 0; p < 4; ++p) nxt[1 + p] = load(col0 + lr + 32 * p, kt * PL_BK + lc);
        };
        auto put = [&](double *dst, const float4 &v) {
            dst[0] = (double)v.x;
            dst[1] = (double)v.y;
            dst[2] = (double)v.z;
            dst[3] = (double)v.w;
        };
        auto store = [&](int buf) {
            put(&sm.As[buf][lr][lc], nxt[0]);
#pragma unroll
            for (int p = 0; p < 4; ++p) put(&sm.Bs[buf][lr + 32 * p][lc], nxt[1 + p]);
        };

        double limit[8];
        uint32_t have[8];  // waiting keys
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            // (a place without a row takes no pairs, as if its tau were 0: its accumulators
            // are some other row's, and under cosine a norm of 0 would let every pair
            // through.  6,000 x 24 cosine, 16 such places: 911 us for the call, 388 now)
            limit[r] = next_limit<METRIC>(sm.rows[warp * 8 + r] == 0xffffffffu ? 0ull : KEY_NONE, sm.rn_a[warp * 8 + r]);
            have[r] = 0;
        }
        fetch(c_begin, 0);
        store(0);
        __syncthreads();

        double acc[8][4];
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[r][c] = 0.0;
        uint32_t col0 = c_begin, kt = 0;
        for (uint32_t s = 0; s < stages; ++s) {
            // the next stage's loads fly while this one is computed
            const bool last_k = kt + 1 == nk;
            const uint32_t ncol = last_k ? col0 + PL_BN : col0, nkt = last_k ? 0u : kt + 1;
            if (s + 1 < stages) fetch(ncol, nkt);
            const int buf = s & 1;
            const double(*A)[PL_BK + 1] = &sm.As[buf][warp * 8];
            const double(*Bm)[PL_BK + 1] = &sm.Bs[buf][lane];
            const int kmax = (int)min((uint32_t)PL_BK, d - kt * PL_BK);
#pragma unroll 4
            for (int kk = 0; kk < kmax; ++kk) {
                double bv[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) bv[c] = Bm[32 * c][kk];
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const double av = A[r][kk];
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[r][c] = pair_step<METRIC>(acc[r][c], av, bv[c]);
                }
            }
            if (last_k) {
                // The first tile of a short list: the k-th smallest of the lanes' own
                // minima bounds the row's k-th distance, so the tile is cut to little
                // more than k pairs before any is merged (cosine's limit is not on
                // the accumulator alone; its first tile is merged as it comes).
                if (KPL == 1 && METRIC != HM_METRIC_COSINE && col0 == c_begin) {
#pragma unroll
                    for (int r = 0; r < 8; ++r) {
                        double mine = __longlong_as_double(0x7ff0000000000000ll);
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            if (col0 + lane + 32 * c < c_end) mine = fmin(mine, acc[r][c]);
                        float f = __double2float_ru(mine);
#pragma unroll
                        for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
                            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                                const float o = __shfl_xor_sync(0xffffffffu, f, stride);
                                f = ((lane & stride) == 0) == ((lane & size) == 0) ? fminf(f, o) : fmaxf(f, o);
                            }
                        const double t = (double)__shfl_sync(0xffffffffu, f, (int)k - 1);
                        if (sm.rows[warp * 8 + r] != 0xffffffffu)
                            limit[r] = pair_limit<METRIC>(pair_finish<METRIC>(t, 0.0, 0.0), 0.0);
                    }
                }
                // pairs that may enter a row's list wait in `fresh`
                double rn_b[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint32_t col = col0 + lane + 32 * c;
                    rn_b[c] = METRIC == HM_METRIC_COSINE && col < c_end ? J.rnorm[col] : 0.0;
                }
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const uint32_t row = sm.rows[warp * 8 + r];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t col = col0 + lane + 32 * c;
                        const double a = acc[r][c];
                        acc[r][c] = 0.0;
                        const bool near = METRIC == HM_METRIC_COSINE ? a >= __dmul_rn(limit[r], rn_b[c]) : a <= limit[r];
                        const bool pass = col < c_end && (near || col == row);
                        const unsigned m = __ballot_sync(0xffffffffu, pass);
                        if (!m) continue;
                        uint64_t *fresh = sm.fresh[warp * 8 + r];
                        if (pass) {
                            float dist = pair_finish<METRIC>(a, sm.rn_a[warp * 8 + r], rn_b[c]);
                            if (col == row) dist = 0.0f;  // src/knn.rs:38-39
                            fresh[have[r] + __popc(m & ((1u << lane) - 1u))] = make_key(dist, col);
                        }
                        have[r] += __popc(m);
                        __syncwarp();
                        if (have[r] >= 32) {
                            limit[r] = plain_merge<METRIC, KPL>(sm.list[warp * 8 + r], fresh, 32, k,
                                                                sm.rn_a[warp * 8 + r]);
                            have[r] -= 32;
                            const uint64_t rest = fresh[32 + lane];
                            __syncwarp();
                            if ((uint32_t)lane < have[r]) fresh[lane] = rest;
                            __syncwarp();
                        }
                    }
                }
            }
            if (s + 1 < stages) store(buf ^ 1);
            col0 = ncol;
            kt = nkt;
            __syncthreads();
        }

        // the first k keys of each row
#pragma unroll 1
        for (int r = 0; r < 8; ++r) {
            uint32_t left = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) left = q == r ? have[q] : left;
            const uint32_t row = sm.rows[warp * 8 + r];
            if (row == 0xffffffffu) continue;
            uint64_t *list = sm.list[warp * 8 + r];
            if (left) plain_merge<METRIC, KPL>(list, sm.fresh[warp * 8 + r], left, k, 0.0);
            for (uint32_t e = lane; e < k; e += 32) {
                const uint64_t key = list[e];
                if (!FALLBACK && J.splits > 1) {
                    J.partial[((size_t)split * (J.q1 - J.q0) + (row - J.q0)) * k + e] = key;
                } else if (FALLBACK && parts > 1) {
                    J.partial[(size_t)row * J.elists * J.cap + split * k + e] = key;
                } else {
                    J.idx[(size_t)row * k + e] = key_idx(key);
                    J.dist[(size_t)row * k + e] = key_dist(key);
                }
            }
        }
        __syncthreads();  // the rows and lists are rewritten by the next group
    }
    if (FALLBACK && parts > 1) merge_parts<KPL>(J, sm, first_grp, parts);
}

template <int METRIC, int KPL, bool FALLBACK>
static int launch_plain_kernel(const PlainWork &w, uint32_t grid, cudaStream_t s) {
    const int smem = (int)sizeof(PlainSmem<KPL>);
    auto *kernel = plain_knn_kernel<METRIC, KPL, FALLBACK>;
    HM_TRY(ensure_dynamic_smem((const void *)kernel, smem));
    HM_CUDA_TRY(launch(true, kernel, grid, PL_THREADS, smem, s, w));
    count_launch();
    return HM_OK;
}
template <int METRIC>
static int launch_plain_metric(const PlainWork &w, uint32_t grid, cudaStream_t s) {
    switch (w.kpl) {
    case 1: return launch_plain_kernel<METRIC, 1, false>(w, grid, s);
    case 2: return launch_plain_kernel<METRIC, 2, false>(w, grid, s);
    case 4: return launch_plain_kernel<METRIC, 4, false>(w, grid, s);
    case 8: return launch_plain_kernel<METRIC, 8, false>(w, grid, s);
    default: return set_error(HM_ERR_UNSUPPORTED, "select width %u", w.kpl);
    }
}
// (the screened paths take k up to 64, and not the manhattan metric)
template <int METRIC>
static int launch_fallback_metric(const PlainWork &w, uint32_t grid, cudaStream_t s) {
    switch (w.kpl) {
    case 1: return launch_plain_kernel<METRIC, 1, true>(w, grid, s);
    case 2: return launch_plain_kernel<METRIC, 2, true>(w, grid, s);
    default: return set_error(HM_ERR_UNSUPPORTED, "select width %u", w.kpl);
    }
}

// One launch per metric present (the arithmetic is a template parameter);
// `w` describes that metric's items or fallback jobs.
int launch_plain(const PlainWork &w, int metric, cudaStream_t s) {
    const uint32_t grid = w.fallback ? w.fb_njobs * w.per_job : w.nitems;
    if (grid == 0) return HM_OK;
    ScopedKernelTimer timer(HM_KCLASS_EXACT, s);
    if (w.fallback) {
        switch (metric) {
        case HM_METRIC_EUCLIDEAN: return launch_fallback_metric<HM_METRIC_EUCLIDEAN>(w, grid, s);
        case HM_METRIC_COSINE: return launch_fallback_metric<HM_METRIC_COSINE>(w, grid, s);
        default: return set_error(HM_ERR_INVALID, "no fallback for metric %d", metric);
        }
    }
    switch (metric) {
    case HM_METRIC_EUCLIDEAN: return launch_plain_metric<HM_METRIC_EUCLIDEAN>(w, grid, s);
    case HM_METRIC_COSINE: return launch_plain_metric<HM_METRIC_COSINE>(w, grid, s);
    case HM_METRIC_MANHATTAN: return launch_plain_metric<HM_METRIC_MANHATTAN>(w, grid, s);
    default: return set_error(HM_ERR_INVALID, "unknown metric %d", metric);
    }
}

// ------------------------------------------------------------ split merge
// One warp per row of an exact-path job with splits > 1 folds its split lists.
template <int KPL>
__global__ void __launch_bounds__(256) merge_splits_kernel(const JobDev *__restrict__ jobs,
                                                           const uint2 *__restrict__ merges, uint32_t nmerges,
                                                           uint32_t rows) {
    grid_ready();
    const int lane = threadIdx.x & 31;
    const uint32_t mr = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (mr >= rows) return;
    uint32_t lo = 0, hi = nmerges;  // the job whose rows hold this one
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (merges[mid].y <= mr) lo = mid; else hi = mid;
    }
    const JobDev &J = jobs[merges[lo].x];
    const uint32_t at = mr - merges[lo].y, row = J.q0 + at, rows_j = J.q1 - J.q0, k = J.k;
    WarpTopK<KPL> top;
#pragma unroll
    for (int q = 0; q < KPL; ++q) {
        const uint32_t e = q * 32 + lane;
        top.v[q] = (e < k) ? J.partial[(size_t)at * k + e] : KEY_NONE;
    }
    top.refresh_tau(k, lane);
    for (uint32_t sp = 1; sp < J.splits; ++sp) {
        const uint64_t *list = J.partial + ((size_t)sp * rows_j + at) * k;
        for (uint32_t e0 = 0; e0 < k; e0 += 32) {
            const uint64_t key = (e0 + lane < k) ? list[e0 + lane] : KEY_NONE;
            if (!__any_sync(0xffffffffu, key < top.tau)) break;  // lists are sorted
            top.template merge32<true>(key, k, lane);
        }
    }
#pragma unroll
    for (int q = 0; q < KPL; ++q) {
        const uint32_t e = q * 32 + lane;
        if (e < k) {
            J.idx[(size_t)row * k + e] = key_idx(top.v[q]);
            J.dist[(size_t)row * k + e] = key_dist(top.v[q]);
        }
    }
}

int launch_merge(const JobDev *jobs, const uint2 *merges, uint32_t nmerges, uint32_t rows, uint32_t kpl,
                 cudaStream_t s) {
    const int blocks = (int)((rows + 7) / 8);
    ScopedKernelTimer timer(HM_KCLASS_SELECT, s);
    auto *merge = kpl == 1   ? merge_splits_kernel<1>
                  : kpl == 2 ? merge_splits_kernel<2>
                  : kpl == 4 ? merge_splits_kernel<4>
                  : kpl == 8 ? merge_splits_kernel<8>
                             : nullptr;
    if (!merge) return set_error(HM_ERR_UNSUPPORTED, "select width %u", kpl);
    HM_CUDA_TRY(launch(true, merge, blocks, 256, 0, s, jobs, merges, nmerges, rows));
    count_launch();
    return HM_OK;
}

}  // namespace hm
