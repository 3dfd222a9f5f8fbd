// hm_internal.cuh -- shared declarations of libholomap_cuda.so.
//
// Numerical contract: every kernel that produces a returned value does so in
// exactly the reference's operation order with explicitly rounded intrinsics
// (__dadd_rn, __dmul_rn, __fadd_rn, ...), and the library is compiled with
// --fmad=false so that nothing is contracted into an FMA.  See the comments in
// each kernel file for the reference lines it follows.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/holomap_cuda.h"

namespace hm {

// ---------------------------------------------------------------- errors
// Thread-local message for hm_last_error(); returns `code` for chaining.
int set_error(int code, const char *fmt, ...);
void clear_error();

#define HM_CUDA_TRY(expr)                                                        \
    do {                                                                         \
        cudaError_t e_ = (expr);                                                 \
        if (e_ != cudaSuccess)                                                   \
            return ::hm::set_error(e_ == cudaErrorMemoryAllocation ? HM_ERR_OOM  \
                                                                   : HM_ERR_CUDA, \
                                   "%s: %s (%s:%d)", #expr, cudaGetErrorString(e_), \
                                   __FILE__, __LINE__);                          \
    } while (0)

#define HM_TRY(expr)              \
    do {                          \
        int rc_ = (expr);         \
        if (rc_ != HM_OK) return rc_; \
    } while (0)

inline size_t round_up(size_t x, size_t m) { return (x + m - 1) / m * m; }

// Kernel launch that may overlap the end of the stream's previous kernel
// (programmatic dependent launch): the blocks become resident while the previous
// kernel's last blocks run and wait in grid_ready(), which every kernel launched
// so calls before anything else.  A kernel starts only when all blocks of the
// previous one have passed their own grid_ready(), so everything but that one
// kernel's output is complete by then: its output must not be read through
// const __restrict__ kernel arguments or __ldg (loads that may move above the
// wait), which here are the job tables, written two or more kernels earlier, and
// the caller's points.  `overlap` false: an ordinary launch.  20,000 x 128 call (17
// launches) 684 -> 656 us, 50,000 x 384 2,717 -> 2,663.  Grids of more than a wave
// of small blocks launch ordinarily: waiting blocks took the slots of the running
// kernel's in the big batch (256 datasets, 540,000 rows: 6,760 us with all grids
// overlapped, 6,648 up to 40,000 blocks, 6,494 up to 2,400).
constexpr uint64_t OVERLAP_BLOCKS = 16 * 148;
template <typename... P, typename... A>
inline cudaError_t launch(bool overlap, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                          A &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    overlap = overlap && (uint64_t)grid.x * grid.y <= OVERLAP_BLOCKS;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
__device__ __forceinline__ void grid_ready() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Sets a kernel's dynamic shared-memory limit once per device (the attribute
// call is kept off the per-launch path).
int ensure_dynamic_smem(const void *func, int bytes);
// Multiprocessor count of the current device (cached; 148 without a device).
int device_sm_count();

// ----------------------------------------------------------- instrumentation
// Every kernel launch calls count_launch(); ScopedKernelTimer records an
// event pair around the launches in its scope when timing is enabled.
void count_launch(uint64_t n = 1);
bool timing_enabled();
void timing_record(int kclass, cudaStream_t s, bool start);

struct ScopedKernelTimer {
    int cls;
    cudaStream_t s;
    bool on;
    ScopedKernelTimer(int c, cudaStream_t st) : cls(c), s(st), on(timing_enabled()) {
        if (on) timing_record(cls, s, true);
    }
    ~ScopedKernelTimer() {
        if (on) timing_record(cls, s, false);
    }
};

// -------------------------------------------------------- composite keys
// Every returned distance is +0.0 or positive (possibly +inf), so its binary32
// bit pattern orders like the value and the 64-bit key (bits << 32) | index
// orders exactly like the reference's (total_cmp(dist), index) sort
// (src/knn.rs:46-48).  ~0 is a sentinel larger than every real key.
constexpr uint64_t KEY_NONE = ~0ull;

__device__ __forceinline__ uint64_t make_key(float dist, uint32_t idx) {
    return ((uint64_t)__float_as_uint(dist) << 32) | (uint64_t)idx;
}
__device__ __forceinline__ float key_dist(uint64_t key) {
    return __uint_as_float((uint32_t)(key >> 32));
}
__device__ __forceinline__ uint32_t key_idx(uint64_t key) { return (uint32_t)key; }

__device__ __forceinline__ uint64_t shfl_u64(uint64_t v, int src) {
    uint32_t lo = __shfl_sync(0xffffffffu, (uint32_t)v, src);
    uint32_t hi = __shfl_sync(0xffffffffu, (uint32_t)(v >> 32), src);
    return ((uint64_t)hi << 32) | lo;
}
__device__ __forceinline__ uint64_t shfl_xor_u64(uint64_t v, int mask) {
    uint32_t lo = __shfl_xor_sync(0xffffffffu, (uint32_t)v, mask);
    uint32_t hi = __shfl_xor_sync(0xffffffffu, (uint32_t)(v >> 32), mask);
    return ((uint64_t)hi << 32) | lo;
}
__device__ __forceinline__ uint64_t shfl_up_u64(uint64_t v, int delta) {
    uint32_t lo = __shfl_up_sync(0xffffffffu, (uint32_t)v, delta);
    uint32_t hi = __shfl_up_sync(0xffffffffu, (uint32_t)(v >> 32), delta);
    return ((uint64_t)hi << 32) | lo;
}

// Bitonic sort, ascending, of 32 * NQ keys, element lane * NQ + q in v[q]: strides
// below NQ stay in the lane.
template <typename K, int NQ>
__device__ __forceinline__ void warp_sort(K (&v)[NQ], uint32_t lane) {
#pragma unroll
    for (uint32_t size = 2; size <= 32 * NQ; size <<= 1) {
#pragma unroll
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= NQ) {
                const uint32_t ls = stride / NQ;
                const bool keep_min = ((lane & ls) == 0) == ((lane & (size / NQ)) == 0);
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    const K o = __shfl_xor_sync(0xffffffffu, v[q], ls);
                    v[q] = keep_min ? min(v[q], o) : max(v[q], o);
                }
            } else {
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    if (q & stride) continue;
                    const K a = min(v[q], v[q | stride]), b = max(v[q], v[q | stride]);
                    const bool up = size < NQ ? (q & size) == 0 : (lane & (size / NQ)) == 0;
                    v[q] = up ? a : b;
                    v[q | stride] = up ? b : a;
                }
            }
        }
    }
}

// A sorted list of the KPL*32 smallest keys seen, spread over a warp: element
// e lives in lane (e % 32) of slot (e / 32).  `tau` is element k-1, the
// admission threshold (warp-uniform).  Insert is warp-collective and requires
// x < tau (so x lands inside the first k elements).
template <int KPL>
struct WarpTopK {
    uint64_t v[KPL];
    uint64_t tau;

    __device__ __forceinline__ void reset() {
#pragma unroll
        for (int q = 0; q < KPL; ++q) v[q] = KEY_NONE;
        tau = KEY_NONE;
    }

    __device__ __forceinline__ void refresh_tau(uint32_t k, int lane) {
        const uint32_t qk = (k - 1) >> 5, lk = (k - 1) & 31;
        uint64_t t = KEY_NONE;
#pragma unroll
        for (int q = 0; q < KPL; ++q)
            if ((uint32_t)q == qk) t = v[q];
        tau = shfl_u64(t, (int)lk);
    }

    __device__ __forceinline__ void insert(uint64_t x, uint32_t k, int lane) {
        int pos = 0;
#pragma unroll
        for (int q = 0; q < KPL; ++q) pos += __popc(__ballot_sync(0xffffffffu, v[q] < x));
        uint64_t carry = KEY_NONE;
#pragma unroll
        for (int q = 0; q < KPL; ++q) {
            uint64_t up = shfl_up_u64(v[q], 1);
            uint64_t last = shfl_u64(v[q], 31);
            if (lane == 0) up = carry;
            const int e = q * 32 + lane;
            v[q] = (e < pos) ? v[q] : (e == pos ? x : up);
            carry = last;
        }
        refresh_tau(k, lane);
    }

    // Merge 32 keys, one per lane (absent ones KEY_NONE), into the list: the batch
    // is sorted (unless it comes so), laid reversed over the list's last 32
    // places, and the smaller of each pair kept, which leaves the list's KPL * 32
    // smallest as one bitonic sequence.
    template <bool SORTED = false>
    __device__ __forceinline__ void merge32(uint64_t b, uint32_t k, int lane) {
        if (!SORTED) b = sort32(b, lane);
        const uint64_t rb = shfl_u64(b, 31 - lane);
        v[KPL - 1] = v[KPL - 1] < rb ? v[KPL - 1] : rb;
#pragma unroll
        for (int stride = KPL / 2; stride > 0; stride >>= 1)
#pragma unroll
            for (int q = 0; q < KPL; ++q)
                if (!(q & stride)) {
                    const uint64_t lo = v[q], hi = v[q | stride];
                    v[q] = lo < hi ? lo : hi;
                    v[q | stride] = lo < hi ? hi : lo;
                }
#pragma unroll
        for (int q = 0; q < KPL; ++q)
#pragma unroll
            for (int stride = 16; stride > 0; stride >>= 1) v[q] = exchange(v[q], stride, true, lane);
        refresh_tau(k, lane);
    }
    // 32 keys, one per lane, ascending
    static __device__ __forceinline__ uint64_t sort32(uint64_t b, int lane) {
#pragma unroll
        for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
            for (int stride = size >> 1; stride > 0; stride >>= 1) b = exchange(b, stride, (lane & size) == 0, lane);
        return b;
    }
    // compare-exchange with lane ^ stride, ascending where `up`
    static __device__ __forceinline__ uint64_t exchange(uint64_t x, int stride, bool up, int lane) {
        const uint64_t o = shfl_xor_u64(x, stride);
        return (((lane & stride) == 0) == up) == (x < o) ? x : o;
    }

    // Offer one key per lane; all lanes' keys below tau are inserted.
    __device__ __forceinline__ void offer(uint64_t key, uint32_t k, int lane) {
        unsigned m = __ballot_sync(0xffffffffu, key < tau);
        while (m) {
            const int src = __ffs(m) - 1;
            const uint64_t x = shfl_u64(key, src);
            insert(x, k, lane);
            m &= m - 1;
            m &= __ballot_sync(0xffffffffu, key < tau);
        }
    }
};

// ------------------------------------------------------------- jobs
// Every kernel works on a table of jobs (independent kNN problems): a single
// call is a batch of one.  Rows of all jobs form one "all-rows" space (job j
// owns rows [arow0, arow0 + n)); screened jobs of one operand format also
// share a "group" row space (job j owns group rows [row0, row0 + n)).

// Device-written counters of one job.
struct JobCounters {
    uint32_t nonfinite_min;  // smallest flat index of a non-finite input, or ~0
    uint32_t zero_count;     // rows whose rho is 0 (global-mean sigma floor)
    uint32_t ovf_count;      // screened rows sent to the exact fallback
    uint32_t max_row;        // most candidates reranked in one row
    unsigned long long candidates;  // candidates reranked exactly
    unsigned long long emitted;     // candidates the screen wrote
    uint32_t band_max_bits;  // widest keep band (binary32 bits)
    uint32_t error_code;     // nonzero if a bounded wait gave up
    uint32_t escalate;       // 1: the job's screen was too coarse for its data; its
                             // split-BF16 copy produced the rows (see JobDev::gate)
    uint32_t escalate_rows;  // rows whose band exceeded the escalation share of tau1
    uint32_t swamped_rows;   // rows with half of their k sampled minima within the band of tau1
    uint32_t csum_done;      // column-sum blocks that have finished
    // screen prep maxima (non-negative doubles as bits): |u|, |e|, |r|,
    // |A row|, |B row|, |u|^2, largest centred |x - mu|^2; then zero rows
    unsigned long long maxb[8];
};

struct JobDev {
    // problem and caller buffers (device pointers)
    uint32_t n, d, k, metric, path;
    uint32_t arow0;  // first row in the all-rows space
    uint32_t q0, q1; // query rows [q0, q1): a row shard; every row is a column
    uint32_t rb0;    // first 128-row screen block of the query rows
    const float *x;
    uint32_t *idx;              // addressed as idx[row * k] for rows in [q0, q1)
    float *dist, *sigma, *rho;  // sigma / rho null: no smooth-kNN
    // exact path (and the screened path's fallback)
    double *rnorm;               // sqrt of the sequential sum of squares (cosine)
    uint32_t splits, split_cols;
    uint64_t *partial;           // splits x (q1 - q0) x k keys (splits > 1); a screened job: its candidate
                                 // lists, elists * cap keys a row, for the fallback's parts
    // smooth-kNN
    double target;               // log2(k), host platform log2
    uint32_t *zero_rows;         // n (before that: finished parts of each group of fallback rows)
    // screened path
    uint32_t group, row0, unit0, kp1, k_steps, k_stages, row_blocks, col_tiles, parts, part_tiles, cap;
    uint32_t seed_tiles;         // leading column tiles of each part in the threshold pass
    // threshold pass: row i's chunk minimum c (c < mins, of 4 << min_shift columns)
    // is minima[min0 + c * min_rows + i]
    unsigned long long min0;
    uint32_t mins, min_shift, min_rows;
    // candidate lists of the emission pass: elists per row (two per column
    // part; with the symmetric emission one more, the row's column list, last)
    uint32_t elists, sym;        // sym: the emission pass covers the tiles on and above the diagonal
    uint32_t erb0, eparts, ept;  // emission units: first row block, column parts per row block, tiles per part
    unsigned long long eslot0;   // first candidate list of the job
    unsigned long long cand0;    // first candidate slot: list l holds [cand0 + (l - eslot0) * cap, +cap)
    float scale;                 // 1 (cosine) or 2 (euclidean)
    double *mu, *csum;           // euclidean column mean and its partial sums
    uint32_t csum_blocks, csum_rows;
    uint32_t *ovf_list;          // n (job-local rows)
    JobCounters *cnt;            // the job's working counters (screen prep maxima)
    JobCounters *out;            // where its reported counts go (the original's for a copy)
    // Escalation: a job screened in BF16 or TF32 may carry a split-BF16 copy
    // (a second job entry on the same points and outputs).  After its
    // threshold pass a kernel decides, from the rows' bands against their
    // thresholds, whether the coarse screen would keep most of the dataset;
    // then the copy runs and the original's remaining kernels step aside.
    // gate: the original's escalate flag (null: always active); the job runs
    // while *gate == gate_on (the original 0, the copy 1).
    const uint32_t *gate;
    uint32_t gate_on;
    uint32_t escalation;         // the original: 1 if it has a copy to hand over to
};

// Whether a job's kernels run: always, unless it takes part in an
// escalation and its side is not the one the flag selects.  The flag is
// written once, between launches (never while a kernel reading it runs).
__device__ __forceinline__ bool job_active(const JobDev &J) {
    return !J.gate || *(volatile const uint32_t *)J.gate == J.gate_on;
}

// Host-side decomposition of an all-rows / item / group index into its job:
// `starts` holds njobs + 1 ascending offsets.
__device__ __forceinline__ uint32_t find_job(const uint32_t *starts, uint32_t njobs, uint32_t idx) {
    uint32_t lo = 0, hi = njobs;  // starts[lo] <= idx < starts[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (starts[mid] <= idx) lo = mid; else hi = mid;
    }
    return lo;
}

int kpl_for_k(uint32_t k);  // 1, 2, 4, 8 or 0 if k > 256

// Rows of padded length K1 at most this take the packed operand kernel
// (several rows per warp); the group's plan records which kernels run.
uint32_t operand_short_k1();
// The autotuner table's path for a problem, (seed_div) the fraction
// 1/seed_div of the columns the screen's threshold pass samples, and whether
// its emission pass takes the symmetric form and the 2-SM form (unless
// hm_tuning_symmetric / hm_tuning_pair force either on this thread).
int autotune_choice(uint64_t n, uint32_t d, uint32_t k, int metric, uint32_t *seed_div, bool *symmetric,
                    bool *pair, bool batched);
// Whether jobs left to the autotuner on the BF16 or TF32 screen carry a
// split-BF16 escalation copy (hm_tuning_escalation).
bool tuning_escalation();

// ------------------------------------------------------------- plain path
constexpr int PL_BM = 32;     // rows per CTA (4 warps x 8 rows)
constexpr int PL_BN = 128;    // columns per tile (32 lanes x 4)
constexpr int PL_BK = 16;     // dimensions per shared-memory stage
constexpr int PL_THREADS = 128;
constexpr uint32_t FB_MAX_PARTS = 32;  // column parts of a group of fallback rows

// Work of the exact path: items (job, group of PL_BM rows, column split); or,
// in fallback mode, each job's overflow list strided over `per_job` CTAs, which
// share its groups by columns where they are few.
struct PlainWork {
    const JobDev *jobs;
    uint32_t njobs;
    const uint2 *items;     // per job of the metric: x = job, y = its first item; item i of a job is
                            // row group q0 / PL_BM + i / splits, split i % splits
    uint32_t nitems, njobs_m;
    uint32_t kpl;           // WarpTopK width for the largest k
    uint32_t fallback;      // 1: rows come from the jobs' overflow lists
    uint32_t per_job;       // fallback: CTAs per job
    const uint32_t *ovf;    // fallback of one job: its count of rows, so that a CTA without any leaves
                            // after one load (null: several jobs)
    const uint32_t *fb_jobs;  // fallback: the jobs that may have overflow rows
    uint32_t fb_njobs;
};

// Zeroes the job counters, checks every input for finiteness and forms the
// cosine row norms (all rows of every job; row_starts / all_rows: the all-rows
// space).
int launch_check(const JobDev *jobs, uint32_t njobs, const uint32_t *row_starts, uint32_t all_rows, cudaStream_t s);

int launch_plain(const PlainWork &w, int metric, cudaStream_t s);

// Device memory of one call on host arrays, with the calling thread's own stream
// to run it on: one block, from the device's stream-ordered pool (which the
// host-array kNN calls fill too, and which keeps what is freed) up to
// CALL_POOL_BYTES, above that allocated and given back by the call itself.  The
// stream is idle when the block is freed.  With cudaMalloc and cudaFree (which wait
// for the device and map its memory anew) a whole fit of 2,000 x 50 on host arrays
// took 3.1 to 3.6 ms, now 1.7.
constexpr size_t CALL_POOL_BYTES = 256ull << 20;
struct CallMemory {
    cudaStream_t s = nullptr;
    char *p = nullptr;
    bool pooled = false;
    int open(size_t bytes);
    ~CallMemory();
};
// merges the split lists of the exact-path jobs with splits > 1: `merges` holds
// (job, first of its rows among the `rows` of the merge)
int launch_merge(const JobDev *jobs, const uint2 *merges, uint32_t nmerges, uint32_t rows, uint32_t kpl,
                 cudaStream_t s);

// ------------------------------------------------------------- smooth kNN
// Per row of every job with smooth-kNN outputs (row_starts: all-rows space);
// rows whose rho is 0 get their unfloored sigma and are listed for the
// job's global-mean floor.
// (overlap false where the job table was written by the kernel just before)
int launch_smooth(const JobDev *jobs, uint32_t njobs, const uint32_t *row_starts, uint32_t rows,
                  uint32_t kmax, cudaStream_t s, bool overlap = true);
// Sequential binary64 mean of each job's n*k distances, applied as the floor
// of its listed rows; one block per job, idle when its list is empty.
int launch_mean_all_floor(const JobDev *jobs, uint32_t njobs, cudaStream_t s);

// batch internals used by the request loop: where a bound batch keeps its
// per-job counters in the workspace, and a job's stats/status from a host
// copy of its counters
size_t batch_counters_offset(const hm_batch *B);
int batch_job_result(const hm_batch *B, uint32_t job, const JobCounters &c, hm_stats *st);
// counters of a finished single-job call (workspace `ws`), read after the
// work queued on `s`; the status is the call's (HM_ERR_INVALID for a
// non-finite input, HM_ERR_TIMEOUT for a bounded wait that gave up)
int single_job_stats(const void *ws, uint64_t n, uint32_t d, uint32_t k, int metric, int path,
                     cudaStream_t s, hm_stats *stats);

}  // namespace hm
