// smooth_knn.cu -- smooth-kNN calibration (rho, sigma) on the device.
//
// Reference: src/smooth_knn.rs:23-80 (per-row rho, 64-step binary32 bisection,
// MIN_K_DIST_SCALE floors), mean at :82-84, and libm::expf reached through
// src/fmath.rs:119-122.
//
// smooth_rows_kernel (k <= 256): G lanes per row (1 to 16), the row in
// registers.  sigma is defined by the bisection's steps, and a step only asks
// on which side of the target the row's sum lies, so most steps are settled
// without the sum itself: a bracket [A, B] around the root with proven margins
// answers every step outside it, and the few steps inside evaluate the sum
// exactly as the reference does.  smooth_knn_kernel: k above 256, one warp per
// row, every step evaluated.  Every evaluated sum is formed in the reference's
// order (j = 1, 2, ..., k-1, each binary32 add rounded) with explicitly rounded
// intrinsics; the file is compiled without FMA contraction or flush-to-zero.
#include <cuda_runtime.h>

#include "hm_internal.cuh"
#include "libm_expf.cuh"

namespace hm {

constexpr uint32_t SK_MAX_K = 256;  // widest row of smooth_rows_kernel
constexpr uint32_t SK_THREADS = 128;  // threads of its blocks

// Row of a thread of smooth_rows_kernel with `lanes` lanes a row.  (The flat thread
// index passes 2^32 from 2^28 rows of 16 lanes on; the rows of a call stay below 2^31.)
__host__ __device__ __forceinline__ uint32_t smooth_row(uint32_t block, uint32_t thread, uint32_t lanes) {
    return block * (SK_THREADS / lanes) + thread / lanes;
}

// One warp per row of the all-rows space; the row's values are read per
// 32-element chunk from global memory (L1 resident after the first pass).
__global__ void __launch_bounds__(256) smooth_knn_kernel(const JobDev *__restrict__ jobs, uint32_t njobs,
                                                         const uint32_t *__restrict__ row_starts,
                                                         uint32_t rows) {
    grid_ready();
    const int lane = threadIdx.x & 31;
    const uint32_t ar = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (ar >= rows) return;
    const JobDev &J = jobs[row_starts ? find_job(row_starts, njobs, ar) : 0];
    if (!J.sigma || !J.rho || J.k <= SK_MAX_K) return;  // smooth_rows_kernel's rows
    const uint32_t row = ar - J.arow0, k = J.k;
    const double target = J.target;
    const float *v = J.dist + (size_t)row * k;
    const uint32_t chunks = (k + 31) / 32;

    // rho: first positive distance in row order, else 0 (src/smooth_knn.rs:35)
    float rh = 0.0f;
    for (uint32_t ch = 0; ch < chunks; ++ch) {
        const uint32_t j = ch * 32 + lane;
        const float x = (j < k) ? v[j] : 0.0f;
        const unsigned m = __ballot_sync(0xffffffffu, x > 0.0f);
        if (m) {
            rh = __shfl_sync(0xffffffffu, x, __ffs(m) - 1);
            break;
        }
    }

    // bisection, binary32 state, hi seeded at f32::MAX (src/smooth_knn.rs:39-65)
    const float f32max = __uint_as_float(0x7f7fffffu);
    float lo = 0.0f, hi = f32max, mid = 1.0f;
    for (int it = 0; it < 64; ++it) {
        float psum = 0.0f;
        for (uint32_t ch = 0; ch < chunks; ++ch) {
            const uint32_t j = ch * 32 + lane;
            float term = 0.0f;
            if (j >= 1 && j < k) {
                const float dd = __fsub_rn(v[j], rh);
                term = (dd > 0.0f) ? expf_libm(-__fdiv_rn(dd, mid)) : 1.0f;
            }
            const uint32_t j_lo = (ch == 0) ? 1u : 0u;
            const uint32_t j_hi = min(32u, k - ch * 32);
            for (uint32_t l = j_lo; l < j_hi; ++l)
                psum = __fadd_rn(psum, __shfl_sync(0xffffffffu, term, (int)l));
        }
        const double ps = (double)psum;
        if (fabs(__dsub_rn(ps, target)) < 1e-5) break;
        if (ps > target) {
            hi = mid;
            mid = __fdiv_rn(__fadd_rn(lo, hi), 2.0f);
        } else {
            lo = mid;
            if (hi >= f32max)
                mid = __fmul_rn(mid, 2.0f);
            else
                mid = __fdiv_rn(__fadd_rn(lo, hi), 2.0f);
        }
    }

    float sg = mid;
    if (rh > 0.0f) {
        // floor = 1e-3 * mean(row), mean = f32(sequential f64 sum / k)
        double s = 0.0;
        for (uint32_t ch = 0; ch < chunks; ++ch) {
            const uint32_t j = ch * 32 + lane;
            const float x = (j < k) ? v[j] : 0.0f;
            const uint32_t j_hi = min(32u, k - ch * 32);
            for (uint32_t l = 0; l < j_hi; ++l)
                s = __dadd_rn(s, (double)__shfl_sync(0xffffffffu, x, (int)l));
        }
        const float mean_row = __double2float_rn(__ddiv_rn(s, (double)k));
        const float floor_v = __fmul_rn(1e-3f, mean_row);
        if (sg < floor_v) sg = floor_v;
    } else if (lane == 0) {
        // floored later with the job's global mean (mean_all_floor_kernel)
        const uint32_t slot = atomicAdd(&J.cnt->zero_count, 1u);
        J.zero_rows[slot] = row;
    }
    if (lane == 0) {
        J.sigma[row] = sg;
        J.rho[row] = rh;
    }
}

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// sum / maximum over the G lanes of a row (every lane of the warp takes part)
template <int G>
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <int G>
__device__ __forceinline__ float row_max(float v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Rows with k_lo < k <= G * NV: lane q of a row holds its values j = G i + q.
//
// With gaps g_j = max(d_j - rho, 0) the row's sum S(mid) = sum_j exp(-g_j / mid)
// is nondecreasing in mid.  Near the target T the reference's binary32 sum psum
// and the quick sum S~ (ex2.approx, any order) lie within
//   |psum - S| <= (k + 2) 2^-24 (T + 1)  (k - 1 rounded adds)
//               + k 2^-23                (the rounded quotient and expf)
//   |S~ - S|   <= 1.3 k 2^-22            (ex2.approx and its rounded argument)
//               + 32 2^-24 (T + 1)       (at most 32 adds a lane and the tree)
// and M is the break tolerance 1e-5 plus 1.1 times their sum.  So S~(B) >= T + M
// proves psum > T + 1e-5 at every mid >= B, S~(A) <= T - M proves psum < T - 1e-5
// at every mid <= A, and the bisection's steps outside (A, B) need no evaluation.
// A and B come from Newton's iteration on c = 1 / mid, where S is convex and
// decreasing: from c = 0 it approaches the root from one side, in 5 to 8 cheap
// evaluations (one ex2 and two multiply-adds a value, no order to keep).  About
// 3 of the bisection's 19 to 40 steps then remain to be evaluated.  Rows outside
// the premises (an infinite gap, gaps beyond 1e+-20) keep A = 0, B = inf: every
// step is evaluated.
//
// What bounds it: instruction issue of the evaluated expf terms and the latency
// of their ordered sum.  Whole calibration, every step evaluated before -> now:
// 1,000 x 15 43 -> 14 us, 50,000 x 30 162 -> 41 us, 150,001 x 15 149 -> 45 us,
// 10,000 x 100 285 -> 45 us.
template <int G, int NV>
__global__ void __launch_bounds__(SK_THREADS, G == 1 ? 4 : 6) smooth_rows_kernel(const JobDev *__restrict__ jobs, uint32_t njobs,
                                                          const uint32_t *__restrict__ row_starts, uint32_t rows,
                                                          uint32_t k_lo) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr float PAD = 1e30f;  // gap of the positions that are not summed: exp(-PAD c) = 0
    grid_ready();
    const int lane = threadIdx.x & 31;
    const uint32_t q = threadIdx.x & (G - 1);
    const uint32_t at = smooth_row(blockIdx.x, threadIdx.x, G);
    const uint32_t ar = min(at, rows - 1);  // lanes past the last row idle along
    const JobDev &J = jobs[row_starts ? find_job(row_starts, njobs, ar) : 0];
    const uint32_t k = J.k;
    const bool mine = at < rows && J.sigma && J.rho && k > k_lo && k <= (uint32_t)(G * NV);
    if (!__any_sync(FULL, mine)) return;
    const uint32_t row = ar - J.arow0;
    const float *src = J.dist + (size_t)row * k;
    float g[NV];  // the values, then the gaps
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const uint32_t j = i * G + q;
        g[i] = mine && j < k ? src[j] : 0.0f;
    }
    // rho: first positive distance in row order, else 0 (src/smooth_knn.rs:35)
    float rh = 0.0f, abs_sum = 0.0f;
    bool found = false;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        abs_sum += fabsf(g[i]);
        if (G == 1) {
            if (!found && g[i] > 0.0f) {
                rh = g[i];
                found = true;
            }
        } else {
            const unsigned m = (__ballot_sync(FULL, g[i] > 0.0f) >> (lane & ~(G - 1))) & ((1u << G) - 1u);
            const float x = __shfl_sync(FULL, g[i], m ? __ffs(m) - 1 : 0, G);
            if (!found && m) {
                rh = x;
                found = true;
            }
        }
    }
    abs_sum = row_sum<G>(abs_sum);
    float zeros = 0.0f, slope = 0.0f, gmax = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const uint32_t j = i * G + q;
        const float dd = __fsub_rn(g[i], rh);
        const bool summed = mine && j >= 1 && j < k;
        g[i] = !summed ? PAD : (dd > 0.0f ? dd : 0.0f);
        if (summed) {
            zeros += g[i] == 0.0f ? 1.0f : 0.0f;
            slope += g[i];
            gmax = fmaxf(gmax, g[i]);
        }
    }
    zeros = row_sum<G>(zeros);
    slope = row_sum<G>(slope);
    gmax = row_max<G>(gmax);

    // the bracket
    const double target = J.target;
    const float T = (float)target, kf = (float)k;
    const float M = 1e-5f + 1.1f * 0x1p-22f * ((0.25f * kf + 8.0f) * (T + 1.0f) + 1.8f * kf);
    const float L2E = 1.44269504f;
    float A = 0.0f, B = __uint_as_float(0x7f800000u);
    const bool newton = mine && k >= 3 && gmax <= 1e20f && gmax >= 1e-20f && zeros < T - M;
    if (zeros >= T + M) B = 0.0f;  // the zero gaps alone exceed the target at every mid
    if (__any_sync(FULL, newton)) {
        float f = kf - 1.0f - T, c = newton ? __fdividef(f, slope) : 1.0f;
        auto eval = [&](float cc, float &S, float &D) {
            const float l = cc * L2E;
            S = 0.0f;
            D = 0.0f;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const float e = ex2_approx(-g[i] * l);
                S += e;
                D += g[i] * e;
            }
            S = row_sum<G>(S);
            D = row_sum<G>(D);
        };
        float S, D;
        for (int it = 0; it < 16; ++it) {
            eval(c, S, D);
            f = S - T;
            const bool more = newton && f > M;
            if (!__any_sync(FULL, more)) break;
            if (more) c += __fdividef(f, D);
        }
        const float cb = c - __fdividef(1.1f * M - f, D), ca = c + __fdividef(1.1f * M + f, D);
        eval(cb, S, D);
        if (newton && cb > 0.0f && S >= T + M) B = __fdiv_rn(1.0f, cb);
        eval(ca, S, D);
        if (newton && ca < 1e30f && S <= T - M) A = __fdiv_rn(1.0f, ca);
    }

    // bisection, binary32 state, hi seeded at f32::MAX (src/smooth_knn.rs:39-65)
    const float f32max = __uint_as_float(0x7f7fffffu);
    float lo = 0.0f, hi = f32max, mid = 1.0f;
    auto advance = [&](bool over) {
        if (over) {
            hi = mid;
            mid = __fmul_rn(__fadd_rn(lo, hi), 0.5f);  // halving rounds as dividing by 2 does
        } else {
            lo = mid;
            mid = hi >= f32max ? __fmul_rn(mid, 2.0f) : __fmul_rn(__fadd_rn(lo, hi), 0.5f);
        }
    };
    int it = mine ? 0 : 64;
    for (;;) {
        while (it < 64 && (mid <= A || mid >= B)) {
            advance(mid >= B);
            ++it;
        }
        __syncwarp();
        if (!__any_sync(FULL, it < 64)) break;
        float psum = 0.0f;
        // gap / mid rounded to binary32: a quotient of two 24-bit numbers lies at
        // least 2^-49 (relative) from every rounding boundary, and the product
        // with the binary64 reciprocal is within 2^-52 of it (below 2^-126, where
        // that fails, exp of either rounding is 1)
        const double inv = __ddiv_rn(1.0, (double)mid);
        auto term_of = [&](float gap) {
            const float e = expf_libm_nonpos(-__double2float_rn(__dmul_rn((double)gap, inv)));
            return gap > 0.0f ? e : 1.0f;
        };
        if (G == 1) {
#pragma unroll
            for (int j = 1; j < NV; ++j) {
                const float t = term_of(g[j]);
                psum = __fadd_rn(psum, j < (int)k ? t : 0.0f);
            }
        } else {
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                // positions that are not summed add +0, which changes nothing
                const float t_i = term_of(g[i]), term = i * G + q < k ? t_i : 0.0f;
#pragma unroll
                for (int s = i == 0 ? 1 : 0; s < G; ++s) psum = __fadd_rn(psum, __shfl_sync(FULL, term, s, G));
            }
        }
        if (it < 64) {
            const double ps = (double)psum;
            if (fabs(__dsub_rn(ps, target)) < 1e-5) {
                it = 64;
            } else {
                advance(ps > target);
                ++it;
            }
        }
    }
    if (!mine) return;
    float sg = mid;
    if (rh > 0.0f) {
        // floor = 1e-3 * mean(row), mean = f32(sequential f64 sum / k); formed
        // only where the row's mean magnitude allows it to matter
        if (q == 0 && !(sg >= 1.001e-3f * __fdividef(abs_sum, kf))) {
            double s = 0.0;
            for (uint32_t j = 0; j < k; ++j) s = __dadd_rn(s, (double)src[j]);
            const float floor_v = __fmul_rn(1e-3f, __double2float_rn(__ddiv_rn(s, (double)k)));
            if (sg < floor_v) sg = floor_v;
        }
    } else if (q == 0) {
        // floored later with the job's global mean (mean_all_floor_kernel)
        const uint32_t slot = atomicAdd(&J.cnt->zero_count, 1u);
        J.zero_rows[slot] = row;
    }
    if (q == 0) {
        J.sigma[row] = sg;
        J.rho[row] = rh;
    }
}

template <int G, int NV>
static int launch_rows(const JobDev *jobs, uint32_t njobs, const uint32_t *row_starts, uint32_t rows, uint32_t k_lo,
                       cudaStream_t s, bool overlap) {
    constexpr uint32_t per_block = SK_THREADS / G;
    HM_CUDA_TRY(launch(overlap, smooth_rows_kernel<G, NV>, (rows + per_block - 1) / per_block, SK_THREADS, 0, s, jobs,
                       njobs, row_starts, rows, k_lo));
    count_launch();
    return HM_OK;
}

int launch_smooth(const JobDev *jobs, uint32_t njobs, const uint32_t *row_starts, uint32_t rows,
                  uint32_t kmax, cudaStream_t s, bool overlap) {
    ScopedKernelTimer timer(HM_KCLASS_SMOOTH, s);
    // Lanes per row: more shorten a row's chain, fewer waste less on shuffles
    // and on waiting for the warp's slowest row.  Measured (whole calibration):
    // k = 15: 5,003 rows 8 lanes 16.4 us, 4 lanes 18.5, 1 lane 22.6; 20,000 rows
    // 20.5 / 18.5 / 20.6; 50,000 rows 34.7 / 28.7 / 24.6.  k = 30: 50,000 rows
    // 45.1 / 41.0 / 66.2.  k = 100, 10,000 rows: 16 lanes 45.0, 32 lanes 49.4.
    if (kmax <= 16) {
        if (rows < 16384) HM_TRY((launch_rows<8, 2>(jobs, njobs, row_starts, rows, 0, s, overlap)));
        else if (rows < 32768) HM_TRY((launch_rows<4, 4>(jobs, njobs, row_starts, rows, 0, s, overlap)));
        else HM_TRY((launch_rows<1, 16>(jobs, njobs, row_starts, rows, 0, s, overlap)));
    } else if (kmax <= 32 || njobs > 1) {
        if (rows < 16384) HM_TRY((launch_rows<8, 4>(jobs, njobs, row_starts, rows, 0, s, overlap)));
        else HM_TRY((launch_rows<4, 8>(jobs, njobs, row_starts, rows, 0, s, overlap)));
    }
    if (kmax > 32 && !(njobs == 1 && kmax > SK_MAX_K)) {
        if (kmax <= 64) HM_TRY((launch_rows<16, 4>(jobs, njobs, row_starts, rows, 32, s, overlap)));
        else if (kmax <= 128) HM_TRY((launch_rows<16, 8>(jobs, njobs, row_starts, rows, 32, s, overlap)));
        else HM_TRY((launch_rows<16, 16>(jobs, njobs, row_starts, rows, 32, s, overlap)));
    }
    if (kmax > SK_MAX_K) {
        HM_CUDA_TRY(launch(overlap, smooth_knn_kernel, (rows + 7) / 8, 256, 0, s, jobs, njobs, row_starts, rows));
        count_launch();
    }
    return HM_OK;
}

// mean_all = f32(sequential binary64 sum of all n*k distances / (n*k))
// (src/smooth_knn.rs:26, :82-84).  The reference's order is one dependent
// chain, so one thread forms it; the other 255 threads of the job's block
// stage the next values through shared memory.  Idle when no row of the job
// had rho == 0.
__global__ void __launch_bounds__(256) mean_all_floor_kernel(const JobDev *__restrict__ jobs) {
    grid_ready();
    const JobDev &J = jobs[blockIdx.x];
    if (!J.sigma || !J.rho) return;
    const uint32_t cnt = J.cnt->zero_count;
    if (cnt == 0) return;
    __shared__ float stage[2][2048];
    __shared__ float floor_v;
    const float *dists = J.dist;
    const uint64_t total = (uint64_t)J.n * J.k;
    double s = 0.0;
    const uint64_t chunk = 2048;
    for (uint64_t base = 0; base < total; base += chunk) {
        const int buf = (int)((base / chunk) & 1);
        const uint64_t len = min(chunk, total - base);
        for (uint64_t t = threadIdx.x; t < len; t += blockDim.x) stage[buf][t] = dists[base + t];
        __syncthreads();
        if (threadIdx.x == 0)
            for (uint64_t t = 0; t < len; ++t) s = __dadd_rn(s, (double)stage[buf][t]);
        // the double buffer lets the next fill overlap the chain; the barrier
        // of the iteration after next protects reuse
    }
    if (threadIdx.x == 0) {
        const float mean_all = __double2float_rn(__ddiv_rn(s, (double)total));
        floor_v = __fmul_rn(1e-3f, mean_all);
    }
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < cnt; t += blockDim.x) {
        const uint32_t row = J.zero_rows[t];
        if (J.sigma[row] < floor_v) J.sigma[row] = floor_v;
    }
}

int launch_mean_all_floor(const JobDev *jobs, uint32_t njobs, cudaStream_t s) {
    ScopedKernelTimer timer(HM_KCLASS_SMOOTH, s);
    HM_CUDA_TRY(launch(true, mean_all_floor_kernel, njobs, 256, 0, s, jobs));
    count_launch();
    return HM_OK;
}

}  // namespace hm

extern "C" uint32_t hm_debug_smooth_row(uint32_t block, uint32_t thread, uint32_t lanes) {
    return hm::smooth_row(block, thread, lanes);
}
