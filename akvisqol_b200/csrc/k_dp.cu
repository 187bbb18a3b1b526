// Patch-alignment DP and backtrack (reference src/dp.zig:216-352).
//
// One CTA per pair. Rows (reference patches) are serial. Within a row the
// CPU keeps a running maximum of the previous row over [prev_lo, slide)
// with `>=` (ties go to the later offset); that is an exclusive prefix scan
// under an associative operator. A thread takes up to eight consecutive slides
// of a row, as few as cover it: it scans them itself, a warp scans its
// threads' totals by shuffles, and every thread adds up the totals of the warps
// before its own (one barrier). Values are compared as integers, and the two
// rows in hand stay in shared memory where they fit. Cells outside a row's
// window are the CPU's zeros: they are not stored but read as such. The
// backtrack is a short serial walk.
//
// Bound by the rows' dependent time. With chunks of 512 slides scanned one
// behind the other, four barriers a chunk, rows in global memory and the table
// cleared first, 16 patches x 497 frames took 44 us and 100 x 2997 1180; now
// 20 and 389. 512 threads take 32 and 460 (barriers), a slide of each round a
// thread 33 and 635 (more scans).
#include <algorithm>

#include "device.cuh"
#include "kernels.h"

namespace vqb {

namespace {

constexpr int kDpThreads = 256;
constexpr int kDpWarps = kDpThreads / 32;
constexpr int kRowsHeld = 12288;  // slides of a row kept in shared memory (two rows, 192 KB)

// A value and its slide, as integers: key orders like the value (zeros alike;
// a NaN, which the CPU's `>=` never takes, is empty like the start).
struct RunMax {
    long long key;
    int32_t i;
};
__device__ constexpr long long kEmpty = -0x7fffffffffffffffll - 1;
__device__ inline RunMax element(double v, int s) {
    const long long b = __double_as_longlong(v + 0.0);
    return v == v ? RunMax{b ^ (b >> 63 & 0x7fffffffffffffffll), s} : RunMax{kEmpty, -1};
}
__device__ inline double value(RunMax x) {  // -inf if empty
    return x.key == kEmpty ? -INFINITY : __longlong_as_double(x.key ^ (x.key >> 63 & 0x7fffffffffffffffll));
}
// Sequential `if (val >= running_max) take` over A then B.
__device__ inline RunMax combine(RunMax a, RunMax b) {
    const bool t = b.key >= a.key;
    return RunMax{t ? b.key : a.key, t ? b.i : a.i};
}
__device__ inline RunMax shfl_up(RunMax x, int off) {
    return RunMax{__shfl_up_sync(0xffffffffu, x.key, off), __shfl_up_sync(0xffffffffu, x.i, off)};
}

// One row of a job: the rows' windows, the previous row's values (slide s at
// prev[s]) and this row's cells.
struct Row {
    int32_t start, end, plo, phi;
    const double *sims, *prev, *next_sims;  // next_sims: the row after's, or null
    double *row;
    int32_t *back;
};

// Slides c0 .. c0 + kPer x kDpThreads - 1, kPer consecutive ones a thread;
// carry: the scan up to c0.
template <int kPer>
__device__ inline void slides(const Row &r, int c0, RunMax &carry, RunMax *totals) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int s0 = c0 + (int)threadIdx.x * kPer;
    double p[kPer], sim[kPer];
    RunMax x{kEmpty, -1}, el[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int s = s0 + k;
        sim[k] = s >= r.start && s <= r.end ? __ldg(r.sims + s) : 0.0;
        p[k] = s <= r.end && s <= r.phi ? r.prev[s] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        el[k] = s0 + k <= r.end ? element(p[k], s0 + k) : RunMax{kEmpty, -1};
        x = combine(x, el[k]);
    }
    if (r.next_sims && s0 <= r.end) asm volatile("prefetch.global.L1 [%0];" ::"l"(r.next_sims + s0));
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const RunMax y = shfl_up(x, off);
        const RunMax z = combine(y, x);
        x.key = lane >= off ? z.key : x.key;
        x.i = lane >= off ? z.i : x.i;
    }
    if (lane == 31) totals[wid] = x;
    RunMax run = shfl_up(x, 1);
    if (lane == 0) run = RunMax{kEmpty, -1};
    __syncthreads();
    // what lies before this warp, and all of it
    RunMax before = carry;
#pragma unroll
    for (int w = 0; w < kDpWarps; ++w) {
        const RunMax t = totals[w];
        if (w < wid) before = combine(before, t);
        carry = combine(carry, t);
    }
    run = combine(before, run);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int s = s0 + k;
        const double moved = sim[k] + value(run);
        const bool stay = p[k] > moved;
        if (s >= r.start && s <= r.end) {
            r.row[s] = stay ? p[k] : moved;
            r.back[s] = stay ? s : run.i;
        }
        run = combine(run, el[k]);
    }
}

// rows_held: slides of the shared-memory rows (0: every row in global memory).
__global__ void __launch_bounds__(kDpThreads) dp_kernel(const DpJob *__restrict__ jobs, int rows_held) {
    extern __shared__ double rows_sm[];  // [2][rows_held]
    const DpJob job = jobs[blockIdx.x];
    const int np = job.np;
    const int64_t cols = job.nf_deg;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    __shared__ RunMax totals[2][kDpWarps];
    __shared__ double best_v[kDpWarps];
    __shared__ int32_t best_i[kDpWarps];

    // slide s of row p is row_at(p, ...)[s]
    auto row_at = [&](int p, int lo, int hi) -> double * {
        return hi - lo < rows_held ? rows_sm + (p & 1) * rows_held - lo : job.dp + (int64_t)p * cols;
    };
    int lo = (int)job.lo[0], hi = (int)job.hi[0];
    Row r;
    r.row = row_at(0, lo, hi);
    for (int s = lo + tid; s <= hi; s += kDpThreads) {
        r.row[s] = job.sims[s];
        job.bt[s] = -1;
    }
    int next_lo = np > 1 ? (int)job.lo[1] : 0, next_hi = np > 1 ? (int)job.hi[1] : 0;
    __syncthreads();
    int par = 0;
    for (int pi = 1; pi < np; ++pi) {
        r.plo = lo, r.phi = hi, r.prev = r.row;
        r.start = lo = next_lo, r.end = hi = next_hi;
        if (pi + 1 < np) next_lo = (int)job.lo[pi + 1], next_hi = (int)job.hi[pi + 1];
        r.sims = job.sims + (int64_t)pi * cols;
        r.next_sims = pi + 1 < np ? r.sims + cols : nullptr;
        r.row = row_at(pi, lo, hi);
        r.back = job.bt + (int64_t)pi * cols;
        RunMax carry{kEmpty, -1};
        // (as few slides a thread as cover the row)
        for (int c0 = r.plo; c0 <= r.end;) {
            const int left = r.end - c0 + 1;
            if (left <= kDpThreads) {
                slides<1>(r, c0, carry, totals[par]);
                c0 += kDpThreads;
            } else if (left <= 2 * kDpThreads) {
                slides<2>(r, c0, carry, totals[par]);
                c0 += 2 * kDpThreads;
            } else if (left <= 4 * kDpThreads) {
                slides<4>(r, c0, carry, totals[par]);
                c0 += 4 * kDpThreads;
            } else {
                slides<8>(r, c0, carry, totals[par]);
                c0 += 8 * kDpThreads;
            }
            par ^= 1;
        }
        __syncthreads();
    }

    // Backtrack from the first maximum of the last row (strict `>`).
    const int last = np - 1;
    struct Best {
        double v;
        int32_t i;
    } best{-INFINITY, 0};
    {
        for (int s = lo + tid; s <= hi; s += kDpThreads)
            if (r.row[s] > best.v) best = Best{r.row[s], s};
    }
    auto first_max = [](Best a, Best b) { return b.v > a.v || (b.v == a.v && b.v > -INFINITY && b.i < a.i) ? b : a; };
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        best = first_max(best, Best{__shfl_xor_sync(0xffffffffu, best.v, off), __shfl_xor_sync(0xffffffffu, best.i, off)});
    if (lane == 0) best_v[wid] = best.v, best_i[wid] = best.i;
    for (int p = tid; p < np; p += kDpThreads) {
        job.offset[p] = -1;
        job.valid[p] = 1;
    }
    __syncthreads();
    if (tid == 0) {
        for (int k = 1; k < kDpWarps; ++k) best = first_max(best, Best{best_v[k], best_i[k]});
        int64_t cur = best.i;
        for (int p = last; p >= 0; --p) {
            job.offset[p] = cur;
            const int64_t back = cur >= job.lo[p] && cur <= job.hi[p] ? job.bt[(int64_t)p * cols + cur] : 0;
            job.valid[p] = back == cur ? 0 : 1;
            if (back < 0) break;
            cur = back;
        }
    }
}

}  // namespace

void launch_dp(const DpJob *d_jobs, int njobs, int64_t max_window, cudaStream_t s) {
    if (njobs <= 0) return;
    const int held = (int)std::min<int64_t>(max_window, kRowsHeld);
    const size_t smem = 2 * (size_t)held * sizeof(double);
    // (the same value from every thread: a smaller one would fail another's launch)
    if (smem > 32 * 1024)
        cudaFuncSetAttribute(dp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             2 * kRowsHeld * (int)sizeof(double));
    dp_kernel<<<njobs, kDpThreads, smem, s>>>(d_jobs, held);
    launch_counter() += 1;
}

}  // namespace vqb
