// screen_prep.cu -- operands and error terms of the tensor-core screen.
//
// For every row i the screen works on a real vector u_i whose inner products
// give the distance ordering exactly:
//   cosine     u_i = x_i / ||x_i||              (c = 1 - u_i.u_j)
//   euclidean  u_i = (x_i - mu) * 2^-s          (c = ||u_i||^2 + ||u_j||^2 - 2 u_i.u_j)
// with mu the column mean and 2^-s a power of two that brings the largest
// ||u_i|| into [0.5, 1) (exact scaling, so no overflow or underflow can arise
// in the screen's binary32 arithmetic).  u_i is formed in binary64, rounded
// to the tensor-core operand format (bf16, tf32, or a bf16 hi/lo split), and
// the exact rounding error of every row is measured in binary64.  The band
// kernel turns those measurements into each row's keep band 2E_i (the
// derivation is in screen.cuh).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "hm_internal.cuh"
#include "screen.cuh"

namespace hm {

constexpr double kFltMin = 1.1754943508222875e-38;  // 2^-126

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void atomic_max_pos(unsigned long long *p, double v) {
    // non-negative doubles order like their bit patterns
    atomicMax(p, (unsigned long long)__double_as_longlong(v));
}

constexpr uint32_t CSUM_BLOCKS = 64;  // column-sum partial blocks per euclidean job
constexpr uint32_t CSUM_THREADS = 512;

// Column means, binary64 (block = job x slice of its rows): the block's threads
// stand side by side over the columns, in as many row strands as fit, eight loads
// in flight each; the job's last block sums the slices' partials.  20,000 x 128:
// 43 us with one strand and a launch of its own for the sum, 19 now (the points
// come from HBM).
__global__ void __launch_bounds__(CSUM_THREADS) column_mean_kernel(const JobDev *__restrict__ jobs,
                                                                   const GroupDev *__restrict__ G) {
    __shared__ double strand_sum[CSUM_THREADS];
    __shared__ uint32_t s_last;
    grid_ready();
    const uint32_t g = blockIdx.x / CSUM_BLOCKS, b = blockIdx.x % CSUM_BLOCKS;
    const JobDev &J = jobs[G->job_ids[g]];
    if (J.metric != HM_METRIC_EUCLIDEAN || !job_active(J)) return;
    // two rounds of loads a slice at least: small jobs of a batch take few slices
    const uint32_t d = J.d, slices = (uint32_t)min((uint64_t)CSUM_BLOCKS, (uint64_t)J.n * d / (16 * CSUM_THREADS) + 1);
    if (b >= slices) return;
    const uint32_t per = (J.n + slices - 1) / slices;
    const uint32_t r0 = min(J.n, b * per), r1 = min(J.n, r0 + per);
    const uint32_t strands = max(1u, CSUM_THREADS / d), strand = d <= CSUM_THREADS ? threadIdx.x / d : 0u;
    for (uint32_t c0 = 0; c0 < d; c0 += CSUM_THREADS) {  // one round up to 512 columns
        const uint32_t c = d <= CSUM_THREADS ? threadIdx.x % d : c0 + threadIdx.x;
        double s = 0.0;
        if (c < d && strand < strands) {
            const float *x = J.x + c;
            uint32_t r = r0 + strand;
            for (; r + 7 * strands < r1; r += 8 * strands) {
                float v[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = x[(size_t)(r + q * strands) * d];
#pragma unroll
                for (int q = 0; q < 8; ++q) s += (double)v[q];
            }
            for (; r < r1; r += strands) s += (double)x[(size_t)r * d];
        }
        if (strands > 1) {
            strand_sum[threadIdx.x] = s;
            __syncthreads();
            if (threadIdx.x < d)
                for (uint32_t q = 1; q < strands; ++q) s += strand_sum[q * d + threadIdx.x];
        }
        if (c < d && strand == 0) J.csum[(size_t)b * d + c] = s;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&J.cnt->csum_done, 1u) == slices - 1 ? 1u : 0u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (uint32_t c = threadIdx.x; c < d; c += CSUM_THREADS) {
        double s = 0.0;
#pragma unroll 16
        for (uint32_t q = 0; q < slices; ++q) s += __ldcg(&J.csum[(size_t)q * d + c]);
        J.mu[c] = s / (double)J.n;
    }
}

// Largest ||x_i - mu||^2 of each euclidean job, for its power-of-two scale.
// A block covers 32 group rows (one job: a job's rows start 32-aligned), a
// warp 4 of them; one atomic per block.
__global__ void __launch_bounds__(256) centred_norm_max_kernel(const JobDev *__restrict__ jobs,
                                                              const GroupDev *__restrict__ G) {
    __shared__ double s_max[8];
    grid_ready();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t gr0 = blockIdx.x * 32;
    const JobDev &J = group_job(jobs, *G, gr0);
    if (J.metric != HM_METRIC_EUCLIDEAN || !job_active(J)) return;  // uniform over the block
    double m = 0.0;
    for (uint32_t r = 0; r < 4; ++r) {
        const uint32_t row = gr0 + warp * 4 + r - J.row0;
        if (row >= J.n) break;  // padding between jobs
        double s = 0.0;
        for (uint32_t t = lane; t < J.d; t += 32) {
            const double v = (double)J.x[(size_t)row * J.d + t] - J.mu[t];
            s += v * v;
        }
        m = fmax(m, warp_sum(s));
    }
    if (lane == 0) s_max[warp] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) m = fmax(m, s_max[w]);
        atomic_max_pos(&J.cnt->maxb[6], m);
    }
}

__device__ __forceinline__ uint16_t to_bf16_bits(double v, double *rounded) {
    const __nv_bfloat16 h = __float2bfloat16_rn((float)v);
    double r = (double)__bfloat162float(h);
    if (fabs(r) < kFltMin) {
        *rounded = 0.0;
        return 0;
    }
    *rounded = r;
    return __bfloat16_as_ushort(h);
}

__device__ __forceinline__ uint32_t to_tf32_bits(double v, double *rounded) {
    uint32_t b;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(b) : "f"((float)v));
    double r = (double)__uint_as_float(b);
    if (fabs(r) < kFltMin) {
        *rounded = 0.0;
        return 0u;
    }
    *rounded = r;
    return b;
}

// Operand rows: the row's elements in the group's format, its binary64 error
// statistics and the additive terms of the screen epilogue.  A row of K1 elements takes 4, 8 or 16 lanes when K1 is at most
// OP_SHORT_K1 (a warp then holds OP_TILE consecutive rows, all loaded before the
// first is worked on), else the warp; each kernel skips the other's jobs.  A lane
// takes 4 consecutive elements at a time, so an operand piece is one 8 or 16 byte
// store.  What it costs besides the traffic is the row's end: its four sums are
// reduced transposed (6 shuffles for the four, each lane left with one of them),
// and the four square roots are one, taken side by side.  A block takes
// consecutive rows, mostly of one job, and combines its warps' maxima before the
// job's counters see them.  256 datasets: 659 us (both kernels) with a
// warp's every lane summing all four, lane 0 taking the roots and 2-byte stores,
// 448 now; 20,000 x 128: 40 -> 25; 50,000 x 384 (BF16): 104 -> 89.
constexpr uint32_t OP_WARPS = 8;
constexpr int OP_BLOCKS_PER_SM = 3;
constexpr uint32_t OP_SHORT_K1 = 64;
constexpr uint32_t OP_TILE = 8;  // short rows a warp holds (in one job, whose rows start 32-aligned)
uint32_t operand_short_k1() { return OP_SHORT_K1; }
constexpr int OP_TF32 = 0, OP_BF16 = 1, OP_SPLIT = 2;

// The column terms past the group's last row (a column tile may reach them).
__device__ __forceinline__ void clear_column_tail(const GroupDev &G) {
    if (blockIdx.x == 0) {
        const uint32_t end = (G.rows + SC_BN - 1) / SC_BN * SC_BN + SC_BN;
        for (uint32_t t = G.rows + threadIdx.x; t < end; t += blockDim.x) G.colterm[t] = 0.0f;
    }
}

template <int MODE, bool SHORT>
__global__ void __launch_bounds__(OP_WARPS * 32, OP_BLOCKS_PER_SM) operand_kernel(const JobDev *__restrict__ jobs,
                                                                                  const GroupDev *__restrict__ Gp) {
    __shared__ double s_max[OP_WARPS][6];
    __shared__ uint32_t s_zero[OP_WARPS];
    __shared__ const JobDev *s_job[OP_WARPS];
    const GroupDev &G = *Gp;
    grid_ready();
    if (group_idle(jobs, G)) return;
    clear_column_tail(G);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    // the job the warp works on: lanes per row, the lane's place in its row, and
    // the sum it is left with (o1, o2: the lane bits that name it): its largest
    // square root so far and, of the first, the sum itself
    const JobDev *cur = nullptr;
    uint32_t lpr = 32, o1 = 16, o2 = 8, zeros = 0;
    double scale = 1.0, top = 0.0, top_sq = 0.0;
    // the maxima over the warp's rows, per sum; lane (value index) writes
    auto maxima = [&](double *out) {
        for (uint32_t o = 16; o > 0; o >>= 1) {
            if (o == o1 || o == o2) continue;
            top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
            top_sq = fmax(top_sq, __shfl_xor_sync(0xffffffffu, top_sq, o));
        }
        const uint32_t v = (lane & o1 ? 2u : 0u) + (lane & o2 ? 1u : 0u);
        if ((lane & ~(int)(o1 | o2)) == 0) {
            out[v] = top;
            if (v == 3) out[4] = top;  // both operand layouts have the same row norm
            if (v == 0) out[5] = top_sq;
        }
        zeros = __reduce_add_sync(0xffffffffu, zeros);
        __syncwarp();
    };
    auto report = [&](const JobDev *J, int from, int to) {  // lane < 6
        double m = 0.0;
        uint32_t z = 0;
        for (int w = from; w < to; ++w) {
            m = fmax(m, s_max[w][lane]);
            z += s_zero[w];
        }
        atomic_max_pos(&J->cnt->maxb[lane], m);
        if (lane == 0 && z) atomicAdd(&J->cnt->maxb[7], (unsigned long long)z);
    };

    const size_t kp = G.kpmax;
    constexpr int STEPS = SHORT ? OP_TILE / 2 : (MODE == OP_SPLIT ? 2 : 4);  // pieces of 4 loaded ahead
    const uint32_t tiles = SHORT ? (G.rows + OP_TILE - 1) / OP_TILE : G.rows;
    // the blocks take chunks of rows in turn (a group's short and long rows lie in
    // runs, of which each kernel works on one kind).  Chunks of one tile a warp
    // against four: short rows of 256 datasets 167 us / 257; of one row against two
    // and eight: their long rows 312 / 281 / 268, 5,003 x 300 26 / 26 / 41
    constexpr uint32_t CHUNK = SHORT ? 1 : 2;  // tiles a warp takes of one
    for (uint32_t i = 0;; ++i) {
        const uint32_t ti = ((i / CHUNK * gridDim.x + blockIdx.x) * CHUNK + i % CHUNK) * OP_WARPS + warp;
        if (i % CHUNK == 0 && ti - warp >= tiles) break;
        if (ti >= tiles) continue;
        const uint32_t gr0 = SHORT ? ti * OP_TILE : ti;
        const JobDev &J = group_job(jobs, G, gr0);
        if (!job_active(J) || (J.kp1 <= OP_SHORT_K1) != SHORT) continue;
        const bool euc = J.metric == HM_METRIC_EUCLIDEAN;
        if (&J != cur) {
            if (cur != nullptr) {
                maxima(s_max[warp]);
                if (lane == 0) s_zero[warp] = zeros;
                __syncwarp();
                if (lane < 6) report(cur, warp, warp + 1);
                __syncwarp();
            }
            cur = &J;
            zeros = 0;
            top = top_sq = 0.0;
            if (SHORT) {
                lpr = J.kp1 > 32 ? 16u : J.kp1 > 16 ? 8u : 4u;
                o1 = lpr >> 1;
                o2 = lpr >> 2;
            }
            scale = 1.0;
            if (euc) {
                const double m = sqrt(__longlong_as_double((long long)J.cnt->maxb[6]));
                if (m > 0.0) {
                    int e;
                    frexp(m, &e);  // m = f * 2^e, f in [0.5, 1)
                    scale = ldexp(1.0, -e);
                }
            }
        }
        const uint32_t d = J.d, kp1 = J.kp1, sl = (uint32_t)lane & (lpr - 1);
        const bool wide = (d & 3) == 0 && (reinterpret_cast<uintptr_t>(J.x) & 15) == 0;
        // four elements from t (0 past the row's end)
        auto load4 = [&](float (&v)[4], const float *xr, uint32_t t, bool real) {
            v[0] = v[1] = v[2] = v[3] = 0.0f;
            if (!real || t >= d) return;
            if (wide) {
                const float4 q = __ldg(reinterpret_cast<const float4 *>(xr + t));
                v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (t + e < d) v[e] = __ldg(xr + t + e);
            }
        };
        double uu, ee, rr, aa;  // the lane's part of the row's sums
        auto piece = [&](const float (&v)[4], uint32_t t, uint32_t gr, bool real, double mul) {
            uint32_t hi4[4], lo4[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                double u = 0.0;
                // cosine rows are scaled by 1 / ||x|| (the operand u is whatever
                // this arithmetic forms: the band is measured from it)
                if (real && t + e < d) u = euc ? ((double)v[e] - __ldg(J.mu + t + e)) * mul : (double)v[e] * mul;
                uu += u * u;
                if (MODE == OP_SPLIT) {
                    double hi, lo;
                    hi4[e] = to_bf16_bits(u, &hi);
                    lo4[e] = to_bf16_bits(u - hi, &lo);
                    const double res = (u - hi) - lo;
                    ee += lo * lo;
                    rr += res * res;
                    aa += 2.0 * hi * hi + lo * lo;
                } else {
                    double r;
                    hi4[e] = MODE == OP_TF32 ? to_tf32_bits(u, &r) : (uint32_t)to_bf16_bits(u, &r);
                    ee += (r - u) * (r - u);
                    aa += r * r;
                }
            }
            if (MODE == OP_TF32) {
                *reinterpret_cast<uint4 *>(static_cast<uint32_t *>(G.opa) + gr * kp + t) =
                    make_uint4(hi4[0], hi4[1], hi4[2], hi4[3]);
                return;
            }
            const uint2 h = make_uint2(hi4[0] | hi4[1] << 16, hi4[2] | hi4[3] << 16);
            uint16_t *A = static_cast<uint16_t *>(G.opa) + gr * kp + t;
            *reinterpret_cast<uint2 *>(A) = h;
            if (MODE == OP_SPLIT) {
                const uint2 l = make_uint2(lo4[0] | lo4[1] << 16, lo4[2] | lo4[3] << 16);
                uint16_t *B = static_cast<uint16_t *>(G.opb) + gr * kp + t;
                *reinterpret_cast<uint2 *>(A + kp1) = h;
                *reinterpret_cast<uint2 *>(A + 2 * kp1) = l;
                *reinterpret_cast<uint2 *>(B) = h;
                *reinterpret_cast<uint2 *>(B + kp1) = l;
                *reinterpret_cast<uint2 *>(B + 2 * kp1) = h;
            }
        };
        auto row_end = [&](uint32_t gr, bool real, bool zero_row) {
            if (MODE == OP_SPLIT && sl == 0) {
                // the last K step's columns past the three segments
                for (uint32_t t = 3 * kp1; t < J.k_steps * 16; t += 8) {
                    *reinterpret_cast<uint4 *>(static_cast<uint16_t *>(G.opa) + gr * kp + t) = make_uint4(0, 0, 0, 0);
                    *reinterpret_cast<uint4 *>(static_cast<uint16_t *>(G.opb) + gr * kp + t) = make_uint4(0, 0, 0, 0);
                }
            }
            const bool h1 = lane & o1, h2 = lane & o2;
            double k0 = (h1 ? rr : uu) + __shfl_xor_sync(0xffffffffu, h1 ? uu : rr, o1);
            double k1 = (h1 ? aa : ee) + __shfl_xor_sync(0xffffffffu, h1 ? ee : aa, o1);
            double v = (h2 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, h2 ? k0 : k1, o2);
            for (uint32_t o = o2 >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const double root = sqrt(v);
            if (!real) {  // padding between jobs: operands of zeros, read only as masked rows and columns
                if (sl == 0) G.colterm[gr] = 0.0f;
                return;
            }
            top = fmax(top, root);
            RowStat &st = G.rowstat[gr];
            if (sl == 0) {
                top_sq = fmax(top_sq, v);
                st.unorm = root;
                st.sqnorm = v;
                const float term = euc ? __double2float_rn(v) : 0.0f;
                G.rowterm[gr] = term;
                G.colterm[gr] = euc ? term : zero_row ? 0.0f : 1.0f;
                G.force[gr] = zero_row ? 1 : 0;
                zeros += zero_row ? 1u : 0u;
            } else if (sl == o2) {
                st.enorm = root;
            } else if (sl == o1) {
                st.rnorm = root;
            } else if (sl == o1 + o2) {
                st.anorm = st.bnorm = root;
            }
        };
        uu = ee = rr = aa = 0.0;
        float xs[STEPS][4];
        if (SHORT) {
            const uint32_t step = 32 / lpr, first = (uint32_t)lane / lpr;
            double rn[STEPS];
#pragma unroll
            for (int q = 0; q < STEPS; ++q) {
                const uint32_t p = q * step + first, row = gr0 + p - J.row0;
                const bool real = p < OP_TILE && row < J.n;
                load4(xs[q], J.x + (size_t)(real ? row : 0u) * d, 4 * sl, real);
                rn[q] = real && !euc ? J.rnorm[row] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < STEPS; ++q) {
                if (q * step >= OP_TILE) break;
                const uint32_t gr = gr0 + q * step + first;
                const bool real = gr - J.row0 < J.n;
                const bool zero_row = !euc && !(rn[q] > 0.0);
                uu = ee = rr = aa = 0.0;
                if (4 * sl < kp1) piece(xs[q], 4 * sl, gr, real, euc ? scale : zero_row ? 0.0 : 1.0 / rn[q]);
                row_end(gr, real, zero_row);
            }
        } else {
            const uint32_t row = gr0 - J.row0;
            const bool real = row < J.n;
            const float *xr = J.x + (size_t)(real ? row : 0u) * d;
            const double rn = real && !euc ? J.rnorm[row] : 0.0;
            const bool zero_row = !euc && !(rn > 0.0);
            const double mul = euc ? scale : zero_row ? 0.0 : 1.0 / rn;
            for (uint32_t t0 = 4 * sl; t0 < kp1; t0 += 128 * STEPS) {
#pragma unroll
                for (int q = 0; q < STEPS; ++q) load4(xs[q], xr, t0 + 128 * q, real);
#pragma unroll
                for (int q = 0; q < STEPS; ++q)
                    if (t0 + 128 * q < kp1) piece(xs[q], t0 + 128 * q, gr0, real, mul);
            }
            __syncwarp();
            row_end(gr0, real, zero_row);
        }
    }
    // the block's maxima: one report per run of warps on the same job
    if (cur != nullptr) maxima(s_max[warp]);
    if (lane == 0) {
        s_zero[warp] = zeros;
        s_job[warp] = cur;
    }
    __syncthreads();
    if (cur == nullptr || lane >= 6 || (warp > 0 && s_job[warp - 1] == cur)) return;
    int end = warp + 1;
    while (end < (int)OP_WARPS && s_job[end] == cur) ++end;
    report(cur, warp, end);
}

// Keep band of one row (binary32 bits, rounded up), written to G.band.
__device__ __forceinline__ uint32_t band_of_row(const JobDev &J, const GroupDev &G, uint32_t gr) {
    const unsigned long long *maxb = J.cnt->maxb;
    const RowStat st = G.rowstat[gr];
    const double Umax = __longlong_as_double((long long)maxb[0]);
    const double Emax = __longlong_as_double((long long)maxb[1]);
    const double Rmax = __longlong_as_double((long long)maxb[2]);
    const double Bmax = __longlong_as_double((long long)maxb[4]);
    const double SQmax = __longlong_as_double((long long)maxb[5]);
    const double K = (double)(G.split ? 3 * J.kp1 : J.kp1);
    const double gam = K * 0x1p-22;  // fp32 accumulation, any summation order
    const double tiny = K * 0x1p-125;
    double eps;
    if (!G.split) {
        eps = st.enorm * Umax + st.unorm * Emax + st.enorm * Emax;
    } else {
        eps = st.enorm * Emax + st.rnorm * Umax + (st.unorm + st.rnorm) * Rmax;
    }
    eps += gam * st.anorm * Bmax + tiny;
    double E;
    if (J.metric == HM_METRIC_EUCLIDEAN)
        E = 2.0 * eps + (st.sqnorm + SQmax) * (0x1p-21 + (double)(J.d + 8) * 0x1p-50);
    else
        E = eps + 0x1p-21 + (double)(J.d + 8) * 0x1p-51;
    const double B = 2.0 * E * (1.0 + 0x1p-10);
    const float bf = __double2float_ru(B);
    G.band[gr] = bf;
    return __float_as_uint(bf);
}

// Keep band 2E_i per row (see screen.cuh for the terms).
__global__ void band_kernel(const JobDev *__restrict__ jobs, const GroupDev *__restrict__ Gp) {
    const GroupDev &G = *Gp;
    grid_ready();
    if (group_idle(jobs, G)) return;
    // a warp's 32 group rows belong to one job (each job's rows start
    // 32-aligned; G.rows is a multiple of 32)
    const uint32_t gr = blockIdx.x * blockDim.x + threadIdx.x;
    if (gr - (threadIdx.x & 31) >= G.rows) return;  // whole warps
    const JobDev &J = group_job(jobs, G, gr);
    if (!job_active(J)) return;  // uniform over the warp (32 rows of one job)
    const bool real = gr < G.rows && gr - J.row0 < J.n;  // not padding between jobs
    uint32_t bits = 0;
    if (real) bits = band_of_row(J, G, gr);
    bits = __reduce_max_sync(0xffffffffu, bits);  // non-negative floats order like their bits
    if ((threadIdx.x & 31) == 0 && bits) atomicMax(&J.out->band_max_bits, bits);
}


__global__ void job_of_kernel(const GroupDev G) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t * 32 < G.rows) G.job_of[t] = G.job_ids[find_job(G.row_starts, G.njobs, t * 32)];
}

int launch_job_of(const GroupDev &G, cudaStream_t s) {
    job_of_kernel<<<(G.rows / 32 + 255) / 256, 256, 0, s>>>(G);
    HM_CUDA_TRY(cudaGetLastError());
    count_launch();
    return HM_OK;
}

int launch_screen_prep(const JobDev *jobs, const GroupDev &G, const GroupDev *Gd, cudaStream_t s) {
    ScopedKernelTimer timer(HM_KCLASS_PREP, s);
    if (G.any_euclidean) {
        HM_CUDA_TRY(launch(true, column_mean_kernel, G.njobs * CSUM_BLOCKS, CSUM_THREADS, 0, s, jobs, Gd));
        // G.rows is a multiple of 32: 32 group rows per block
        HM_CUDA_TRY(launch(true, centred_norm_max_kernel, G.rows / 32, 256, 0, s, jobs, Gd));
        count_launch(2);
    }
    const uint32_t op_cap = (uint32_t)device_sm_count() * OP_BLOCKS_PER_SM;
    auto both = [&](auto rows_kernel, auto short_rows_kernel) {
        const uint32_t row_blocks = (G.rows + OP_WARPS - 1) / OP_WARPS;
        const uint32_t tile_blocks = (G.rows + OP_WARPS * OP_TILE - 1) / (OP_WARPS * OP_TILE);
        cudaError_t e = cudaSuccess;
        if (G.any_long_rows)
            e = launch(true, rows_kernel, row_blocks < op_cap ? row_blocks : op_cap, OP_WARPS * 32, 0, s, jobs, Gd);
        if (e == cudaSuccess && G.any_short_rows)
            e = launch(true, short_rows_kernel, tile_blocks < op_cap ? tile_blocks : op_cap, OP_WARPS * 32, 0, s, jobs, Gd);
        return e;
    };
    cudaError_t err;
    if (G.kind == SCREEN_KIND_TF32)
        err = both(operand_kernel<OP_TF32, false>, operand_kernel<OP_TF32, true>);
    else if (!G.split)
        err = both(operand_kernel<OP_BF16, false>, operand_kernel<OP_BF16, true>);
    else
        err = both(operand_kernel<OP_SPLIT, false>, operand_kernel<OP_SPLIT, true>);
    HM_CUDA_TRY(err);
    count_launch((G.any_long_rows ? 1 : 0) + (G.any_short_rows ? 1 : 0));
    return HM_OK;
}

int launch_screen_band(const JobDev *jobs, const GroupDev &G, const GroupDev *Gd, cudaStream_t s) {
    ScopedKernelTimer timer(HM_KCLASS_PREP, s);
    HM_CUDA_TRY(launch(true, band_kernel, (G.rows + 255) / 256, 256, 0, s, jobs, Gd));
    count_launch();
    return HM_OK;
}

}  // namespace hm
