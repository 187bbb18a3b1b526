// Exact form: a signal's sums in the CPU's order, s_{k+1} = fl(s_k + t_k)
// from +0, every rounding of the left-to-right loop reproduced (reference
// src/envelope.zig:28-41, src/audio.zig:132-136), without running the chain
// of dependent additions from end to end.
//
// The terms are cut into segments that are simulated side by side from
// guessed starting sums, and the true sums are then threaded through them:
//
//   1. parts: each segment's approximate sums (trees, any rounding).
//   2. bounds, spec: a segment's starting sum is known to within the rounding
//      errors accumulated before it, some thousands of ulps. One lane runs the
//      segment's additions from the approximate start with its low three
//      bits replaced by r, for each r in 0..7, and records the end, and how
//      far the true start may lie from this one for the run to stay valid.
//   3. resolve: from s = 0 on, each segment's lane with the true start's low
//      bits gives the next true sum: end + (s - start).
//
// Why that is exact. Let v_i be a lane's sums and v'_i the true ones, with
// v'_0 = v_0 + d. If v_i + t_i and v_i + t_i + d lie inside one binade with
// spacing u and d is a multiple of 2u, both round to the same side (ties
// too: d keeps the parity), so v'_{i+1} = v_{i+1} + d. The lane keeps
// the largest exponent its sums reach (2u of it must divide d; equal low
// bits make d a multiple of eight starting ulps, so the sums may reach two
// binades above the start, and the start is taken where the approximate sum
// is largest in a 64-sample window to stay within that) and the smallest
// distance of a sum from its binade's ends (which must cover |d| and the
// rounding). d = 0 needs no condition: the lane's run is the true one.
//
// A segment that fails its conditions is still predicted by end + d, which
// is nearly always right (16-bit samples put alternating sums next to powers
// of two, where the distance alone cannot tell); the predictions of 128
// segments are checked at once, a thread adding each doubtful segment term by
// term from its predicted start, and the walk restarts behind the first that
// differs. Infinities, NaN and sums near the subnormals fail the
// conditions and take that path.
//
// The chain bounds such a sum: one dependent f64 add a sample, 10 cycles each
// when run from end to end (before, with one warp per signal and integer tiles
// for the sums of x and x*x, 480,000 samples took 0.75 ms for both, 1.3 ms for
// the alternating sum and 0.7 ms for the aligned energy). Now a segment's
// simulation (20 cycles a sample: nine instructions of one warp, which shares
// its scheduler with at most one other) and the walk (66 cycles a segment)
// take 14 us each for 480,000 samples; the alternating sum takes them twice.
#include <algorithm>
#include <type_traits>

#include "device.cuh"
#include "kernels.h"

namespace vqb {

namespace {

enum SumKind : int {
    kSum = 0,      // sum x
    kEnergy = 1,   // sum x*x
    kNyquist = 2,  // sum (-1)^k (x - sum x / len)
};

constexpr int kVar = 8;        // simulated starts per segment
constexpr int kSegs = 32 / kVar;  // segments per warp
constexpr int kWarps = 4;      // warps per spec CTA
constexpr int kTile = 64;      // samples of a segment staged at a time
constexpr int kRow = kTile + 2;  // a segment's row in a stage (four rows in different banks)
constexpr int kStages = 4;
constexpr int kBatch = 128;    // segments resolve walks at a time, one of its threads each

// One segment's approximate sums over [j L, (j+1) L).
struct Part {
    double s[3];       // x, x*x, (-1)^k x
    int64_t first_nz;  // first k with x*x != 0, or the signal's length
};

// A job's segment records: two chains' arrays of `cap` segments.
struct Chains {
    Part *parts;      // [jobs][cap]
    int64_t *pos;     // [jobs][2][cap + 1]: first term of each segment
    int64_t *start;   // [jobs][2][cap]: bits of the guessed start, low three zero
    double *end;      // [jobs][2][cap][kVar]
    double *slack;    // [jobs][2][cap][kVar]: largest |d| a run is valid for, or -1
};

// The samples a job sums: sample(k), k < len. False: nothing to do.
__device__ inline bool job_signal(const SumJob &job, VSig &sig, double *&out) {
    sig = job.sig;
    out = job.out;
    return true;
}
// The lag-aligned degraded signal drops its first `skip` samples. Its sum is
// the whole signal's when every dropped term is zero: the whole-signal chain
// holds +0 through them and then adds the same terms in the same order.
// Delays, whose dropped samples are the prepended silence, take this path.
__device__ inline bool job_signal(const AlignedEnergyJob &job, VSig &sig, double *&out) {
    int64_t skip, alen;
    aligned_range(job, skip, alen);
    sig = VSig{job.deg.base, job.deg.head - skip, job.deg.avail, job.deg.len - skip};
    out = job.out;
    const bool whole = job.deg_stats && (double)skip <= job.deg_stats[3];
    if (blockIdx.x == 0 && blockIdx.z == 0 && threadIdx.x == 0) {
        out[1] = (double)alen;
        if (whole) out[0] = job.deg_stats[2];
    }
    return !whole;
}

// Where a kind's sum goes: SumJob out[0] = sum x, out[1] = the alternating
// sum, out[2] = sum x*x; an aligned energy's is out[0].
__device__ inline int out_slot(const SumJob &, int kind) { return kind == kSum ? 0 : kind == kNyquist ? 1 : 2; }
__device__ inline int out_slot(const AlignedEnergyJob &, int) { return 0; }

template <int KIND>
__device__ inline double term(double x, int64_t k, double mean) {
    if (KIND == kSum) return x;
    if (KIND == kEnergy) return x * x;
    const double d = x - mean;
    return (k & 1) ? -d : d;
}

// The mean kNyquist subtracts (its sum already in out[0]).
template <int KIND>
__device__ inline double mean_of(const double *out, int64_t len) {
    return KIND == kNyquist ? out[0] / (double)len : 0.0;
}

// ---- 1: approximate sums of the segments, a warp each -----------------------
template <class Job>
__global__ void __launch_bounds__(256) parts_kernel(const Job *__restrict__ jobs, Part *__restrict__ parts, int cap,
                                                    int L) {
    VSig sig;
    double *out;
    if (!job_signal(jobs[blockIdx.y], sig, out)) return;
    const int lane = threadIdx.x & 31;
    const int64_t j = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (j * L >= sig.len) return;
    const int64_t end = (j + 1) * L < sig.len ? (j + 1) * L : sig.len;
    double s = 0.0, e = 0.0, a = 0.0;
    int64_t nz = sig.len;
#pragma unroll 8
    for (int64_t k = j * L + lane; k < end; k += 32) {
        const double x = vsig_at(sig, k);
        s += x;
        e += x * x;
        a += (k & 1) ? -x : x;
        if (x * x != 0.0 && k < nz) nz = k;
    }
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        e += __shfl_xor_sync(0xffffffffu, e, o);
        a += __shfl_xor_sync(0xffffffffu, a, o);
        const int64_t other = __shfl_xor_sync(0xffffffffu, nz, o);
        nz = other < nz ? other : nz;
    }
    if (lane == 0) parts[(int64_t)blockIdx.y * cap + j] = Part{{s, e, a}, nz};
}

// ---- 2: the segments from guessed starts ---------------------------------------

// Segment j's first term and its approximate starting sum: of the 64 terms
// from j L on, the one before which the sum is largest in magnitude (to 14
// bits; ties to the first). The start is marked (low bit) to be simulated. A
// warp per segment.
template <class Job, int KIND0>
__global__ void __launch_bounds__(128) bounds_kernel(const Job *__restrict__ jobs, Chains ch, int cap, int L) {
    VSig sig;
    double *out;
    if (!job_signal(jobs[blockIdx.y], sig, out)) return;
    const int lane = threadIdx.x & 31;
    const int kind = KIND0 == kSum && blockIdx.z == 1 ? kEnergy : KIND0;
    const int64_t nseg = (sig.len + L - 1) / L, j = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (j >= nseg) return;
    const int64_t c = (int64_t)blockIdx.y * 2 + blockIdx.z, k = j * L + 2 * lane;
    const double mean = mean_of<KIND0>(out, sig.len);
    const double *parts = ch.parts[(int64_t)blockIdx.y * cap].s + kind;
    auto term_at = [&](int64_t i) {
        const double x = vsig_at(sig, i);
        return kind == kSum ? x : kind == kEnergy ? x * x : term<kNyquist>(x, i, mean);
    };
    const double t0 = k < sig.len ? term_at(k) : 0.0, t1 = k + 1 < sig.len ? term_at(k + 1) : 0.0;
    double before = 0.0, incl = t0 + t1;
#pragma unroll 4
    for (int64_t i = lane; i < j; i += 32) before += parts[i * (int64_t)(sizeof(Part) / sizeof(double))];
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    double excl = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) excl = 0.0;
    const double v0 = before + excl, v1 = v0 + t0;
    // (the high word's leading bits, then the earlier position)
    const unsigned m0 = k < sig.len ? (__double2hiint(v0) & 0x7fffffc0u) | (63 - 2 * lane) : 0;
    const unsigned m1 = k + 1 < sig.len ? (__double2hiint(v1) & 0x7fffffc0u) | (62 - 2 * lane) : 0;
    const int p = 63 - (int)(__reduce_max_sync(0xffffffffu, m0 > m1 ? m0 : m1) & 63);
    if (lane == p >> 1) {
        const double g = j == 0 ? 0.0 : p & 1 ? v1 : v0;
        ch.pos[c * (cap + 1) + j] = j == 0 ? 0 : j * L + p;
        ch.start[c * cap + j] = (__double_as_longlong(g) & ~(long long)(kVar - 1)) | 1;
        if (j == nseg - 1) ch.pos[c * (cap + 1) + nseg] = sig.len;
    }
}

// 8-byte asynchronous copy to shared memory; `in` false writes zeros (src
// must still be a global address).
__device__ inline void copy8(double *dst, const double *src, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(in ? 8 : 0) : "memory");
}

// The marked segments' runs; the marks are taken off.
template <int KIND>
__device__ inline void spec(const VSig &sig, double mean, const int64_t *__restrict__ pos_in,
                            int64_t *__restrict__ start, double *__restrict__ end_out,
                            double *__restrict__ slack_out, int L, double *__restrict__ stages) {
    const int lane = threadIdx.x & 31, mine = lane / kVar, r = lane % kVar;
    const int64_t nseg = (sig.len + L - 1) / L;
    const int64_t j0 = ((int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5)) * kSegs, j = j0 + mine;
    if (j0 >= nseg) return;
    const long long at = j < nseg ? start[j] : 0;
    const bool marked = (at & 1) != 0;
    if (!__any_sync(0xffffffffu, marked)) return;
    int64_t pos[kSegs + 1];
#pragma unroll
    for (int b = 0; b <= kSegs; ++b) pos[b] = pos_in[j0 + b < nseg ? j0 + b : nseg];
    int64_t a = 0, b = 0;
#pragma unroll
    for (int q = 0; q < kSegs; ++q)
        if (q == mine) a = pos[q], b = pos[q + 1];
    const long long base = at & ~(long long)(kVar - 1);
    double v = __longlong_as_double(base | r);
    // of |v|: the smallest and largest high words, and of its leading 32
    // mantissa bits the smallest and largest (how near a binade's ends)
    unsigned top = 0, bottom = 0x7fffffffu, frac_min = 0xffffffffu, frac_max = 0;
    const int steps = (int)__reduce_max_sync(0xffffffffu, (unsigned)(b - a));
    const int ntiles = (steps + kTile - 1) / kTile;
    auto issue = [&](int t) {
        if (t < ntiles) {
            double *st = stages + (t % kStages) * kSegs * kRow;
#pragma unroll
            for (int c = 0; c < kSegs * kTile / 32; ++c) {
                const int q = c * 32 / kTile, i = c * 32 % kTile + lane;
                const int64_t k = pos[q] + (int64_t)t * kTile + i, x = k - sig.head;
                const bool in = k < pos[q + 1] && (uint64_t)x < (uint64_t)sig.avail;
                copy8(st + q * kRow + i, in ? sig.base + x : end_out, in);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    const int odd = (int)(a & 1);
    auto add = [&](double x, int i) {
        double t = KIND == kEnergy ? x * x : x;
        if (KIND == kNyquist) {
            t = x - mean;
            t = ((odd ^ i) & 1) ? -t : t;
        }
        return v + t;
    };
    auto look = [&](double w0, double w1) {
        const unsigned h0 = __double2hiint(w0), h1 = __double2hiint(w1);
        const unsigned f0 = __funnelshift_l(__double2loint(w0), h0, 12), f1 = __funnelshift_l(__double2loint(w1), h1, 12);
        top = __vimax3_u32(top, h0 & 0x7fffffffu, h1 & 0x7fffffffu);
        bottom = __vimin3_u32(bottom, h0 & 0x7fffffffu, h1 & 0x7fffffffu);
        frac_min = __vimin3_u32(frac_min, f0, f1);
        frac_max = __vimax3_u32(frac_max, f0, f1);
    };
#pragma unroll
    for (int t = 0; t < kStages - 1; ++t) issue(t);
    // sixteen additions, and beside them the looks at the sixteen before, so
    // that the chain of additions is all that a step waits for
    constexpr int kStep = 16;
    double seen[kStep];
#pragma unroll
    for (int i = 0; i < kStep; ++i) seen[i] = v;
    for (int t = 0; t < ntiles; ++t) {
        issue(t + kStages - 1);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 1) : "memory");
        __syncwarp();
        const double *st = stages + ((t % kStages) * kSegs + mine) * kRow;
        const int left = (int)(b - a) - t * kTile;  // (lanes without a segment just run along)
        auto tile = [&](auto whole) {
#pragma unroll 2
            for (int c = 0; c < kTile; c += kStep) {
                double now[kStep];
#pragma unroll
                for (int i = 0; i < kStep; i += 2) {
                    const double2 x = *reinterpret_cast<const double2 *>(st + c + i);
                    const double w0 = add(x.x, i);
                    v = decltype(whole)::value || c + i < left ? w0 : v;
                    now[i] = v;
                    const double w1 = add(x.y, i + 1);
                    v = decltype(whole)::value || c + i + 1 < left ? w1 : v;
                    now[i + 1] = v;
                    look(seen[i], seen[i + 1]);
                }
#pragma unroll
                for (int i = 0; i < kStep; ++i) seen[i] = now[i];
            }
        };
        if (__all_sync(0xffffffffu, left >= kTile || !marked))
            tile(std::true_type{});
        else
            tile(std::false_type{});
        __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < kStep; i += 2) look(seen[i], seen[i + 1]);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    if (!marked) return;
    // A sum's distance from the ends of its binade [2^e, 2^(e+1)): at least
    // min(frac, 2^32 - 1 - frac) 2^(e-32). 2u of the largest binade comes off
    // it for the rounding.
    const int e0 = (int)((base >> 52) & 0x7ff), etop = max((int)(top >> 20), e0), ebot = (int)(bottom >> 20);
    const unsigned frac = min(frac_min, 0xffffffffu - frac_max);
    double slack = -1.0;
    if (e0 >= 60 && ebot >= 60 && etop < 0x7ff && etop + 1 <= e0 + 3)
        slack = __dsub_rd((double)frac * __hiloint2double((ebot - 32) << 20, 0), __hiloint2double((etop - 51) << 20, 0));
    end_out[j * kVar + r] = v;
    slack_out[j * kVar + r] = slack;
    if (r == 0) start[j] = base;
}

// grid (spec CTAs, jobs, chains): a warp simulates four segments of a chain,
// eight lanes each.
template <class Job, int KIND0>
__global__ void __launch_bounds__(32 * kWarps) spec_kernel(const Job *__restrict__ jobs, Chains ch, int cap, int L) {
    __shared__ __align__(16) double stages[kWarps][kStages * kSegs * kRow];
    VSig sig;
    double *out;
    if (!job_signal(jobs[blockIdx.y], sig, out)) return;
    const int64_t c = (int64_t)blockIdx.y * 2 + blockIdx.z;
    const int64_t *pos = ch.pos + c * (cap + 1);
    int64_t *start = ch.start + c * cap;
    double *end = ch.end + c * cap * kVar, *slack = ch.slack + c * cap * kVar, *st = stages[threadIdx.x >> 5];
    if (KIND0 == kSum && blockIdx.z == 1)
        spec<kEnergy>(sig, 0.0, pos, start, end, slack, L, st);
    else
        spec<KIND0>(sig, mean_of<KIND0>(out, sig.len), pos, start, end, slack, L, st);
}

// ---- 3: the true sums through the segments ---------------------------------

__device__ inline void copy16(void *dst, const void *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

struct ResolveStage {
    double end[kBatch * kVar], slack[kBatch * kVar];
    int64_t start[kBatch];
};

// DRAFT: the walk alone, without checks: a segment whose conditions fail is
// given the start the walk predicts and marked (low bit), to be simulated
// again from there.
template <int KIND, bool DRAFT>
__device__ inline double resolve(const VSig &sig, double mean, const int64_t *__restrict__ pos,
                                 int64_t *__restrict__ start, const double *__restrict__ end,
                                 const double *__restrict__ slack, int L, ResolveStage *stage) {
    __shared__ double walk[kBatch + 1];  // the sum each segment of the batch starts from
    __shared__ int first_bad;
    const int64_t nseg = (sig.len + L - 1) / L;
    auto fetch = [&](int64_t j0, ResolveStage &st) {
        const int n = (int)(nseg - j0 < kBatch ? nseg - j0 : kBatch);
        for (int e = threadIdx.x; e < n * kVar / 2; e += blockDim.x) {
            copy16(st.end + 2 * e, end + j0 * kVar + 2 * e);
            copy16(st.slack + 2 * e, slack + j0 * kVar + 2 * e);
        }
        for (int e = threadIdx.x; 2 * e < n; e += blockDim.x) copy16(st.start + 2 * e, start + j0 + 2 * e);
    };
    double s = 0.0;
    fetch(0, stage[0]);
    for (int64_t j0 = 0; j0 < nseg; j0 += kBatch) {
        const ResolveStage &st = stage[(j0 / kBatch) & 1];
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        if (j0 + kBatch < nseg) fetch(j0 + kBatch, stage[(j0 / kBatch + 1) & 1]);
        const int count = (int)(nseg - j0 < kBatch ? nseg - j0 : kBatch), mine = threadIdx.x;
        int from = 0;
        for (;;) {
            // the walk, every condition taken to hold (no branch waits on a
            // sum), the same in every lane of warp 0
            if (threadIdx.x < 32) {
                double w = s;
#pragma unroll 4
                for (int j = from; j < count; ++j) {
                    const int r = (int)(__double_as_longlong(w) & (kVar - 1));
                    const double d = w - __longlong_as_double(st.start[j] | r);
                    if (threadIdx.x == 0) walk[j] = w;
                    w = st.end[j * kVar + r] + d;
                }
                if (threadIdx.x == 0) walk[count] = w, first_bad = kBatch;
            }
            __syncthreads();
            // the segments whose conditions fail, a thread each, term by term
            double v = 0.0;
            if (mine >= from && mine < count) {
                v = walk[mine];
                const long long sb = __double_as_longlong(v), base = st.start[mine];
                const int r = (int)(sb & (kVar - 1));
                const double d = v - __longlong_as_double(base | r);
                const bool holds = d == 0.0 || (((sb ^ base) >> 52) == 0 && fabs(d) <= st.slack[mine * kVar + r]);
                if (DRAFT) {
                    if (!holds) start[j0 + mine] = (sb & ~(long long)(kVar - 1)) | 1;
                } else if (!holds) {
                    const int64_t a = pos[j0 + mine], b = pos[j0 + mine + 1];
                    constexpr int kAhead = 32;
                    for (int64_t k = a; k < b && v == v; k += kAhead) {  // (a NaN sum stays NaN)
                        double t[kAhead];
#pragma unroll
                        for (int i = 0; i < kAhead; ++i) t[i] = k + i < b ? vsig_at(sig, k + i) : 0.0;
                        // (past the end: +0 leaves any sum that started at +0 as it is)
#pragma unroll
                        for (int i = 0; i < kAhead; ++i) v += k + i < b ? term<KIND>(t[i], k + i, mean) : 0.0;
                    }
                    const double told = walk[mine + 1];
                    if (__double_as_longlong(v) != __double_as_longlong(told) && (v == v || told == told))
                        atomicMin(&first_bad, mine);
                }
            }
            __syncthreads();
            const int bad = first_bad;
            if (bad == kBatch) break;
            __syncthreads();
            if (mine == bad) walk[bad + 1] = v;
            __syncthreads();
            s = walk[bad + 1];
            from = bad + 1;
            if (from >= count || s != s) {
                __syncthreads();
                if (mine == 0) walk[count] = s;
                __syncthreads();
                break;
            }
        }
        s = walk[count];
        __syncthreads();
        if (s != s) break;  // a NaN sum stays NaN
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    return s;
}

// One CTA per (job, chain); the walk's step is two dependent f64 adds and a
// shared-memory read.
template <class Job, int KIND0, bool DRAFT>
__global__ void __launch_bounds__(kBatch) resolve_kernel(const Job *__restrict__ jobs, Chains ch, int cap, int L) {
    __shared__ __align__(16) ResolveStage stage[2];
    VSig sig;
    double *out;
    if (!job_signal(jobs[blockIdx.y], sig, out)) return;
    const int64_t c = (int64_t)blockIdx.y * 2 + blockIdx.z;
    const Part *parts = ch.parts + (int64_t)blockIdx.y * cap;
    const int64_t *pos = ch.pos + c * (cap + 1);
    int64_t *start = ch.start + c * cap;
    const double *end = ch.end + c * cap * kVar, *slack = ch.slack + c * cap * kVar;
    constexpr bool kBoth = KIND0 == kSum;
    double s;
    if (kBoth && blockIdx.z == 1)
        s = resolve<kEnergy, DRAFT>(sig, 0.0, pos, start, end, slack, L, stage);
    else
        s = resolve<KIND0, DRAFT>(sig, mean_of<KIND0>(out, sig.len), pos, start, end, slack, L, stage);
    if (DRAFT) return;
    if (threadIdx.x == 0) out[out_slot(jobs[blockIdx.y], kBoth && blockIdx.z == 1 ? kEnergy : KIND0)] = s;
    if (kBoth && blockIdx.z == 1 && threadIdx.x < 32) {
        // out[3]: the first index with a nonzero energy term (len if none)
        int64_t nz = sig.len;
        for (int64_t j = threadIdx.x; j * L < sig.len; j += 32) nz = parts[j].first_nz < nz ? parts[j].first_nz : nz;
        for (int o = 16; o > 0; o >>= 1) {
            const int64_t other = __shfl_xor_sync(0xffffffffu, nz, o);
            nz = other < nz ? other : nz;
        }
        if (threadIdx.x == 0) out[3] = (double)nz;
    }
}

// Samples a segment: the walk costs 66 cycles a segment, the simulation 20 a
// sample, so their sum is least near L = 1.8 sqrt(n) (480,000 samples: 14 + 14
// us at 1024).
int segment_length(int64_t max_len) {
    return max_len < (1 << 16) ? 256 : max_len < (1 << 18) ? 512 : max_len < (1 << 21) ? 1024 : 2048;
}

// Segment records a job has room for (one more than its segments, even: they
// are read in 16-byte pieces).
int segment_cap(int64_t max_len) {
    const int L = segment_length(max_len);
    return (int)((max_len + L - 1) / L / 2 * 2 + 2);
}

size_t job_scratch(int cap) { return (size_t)cap * sizeof(Part) + 2 * (size_t)(cap + 1) * 8 + 2 * (size_t)cap * (8 + 2 * kVar * 8); }

// Jobs a launch takes: the scratch of one launch is used again by the next.
int jobs_per_launch(int cap) { return (int)std::min<size_t>(16384, std::max<size_t>(1, (size_t(64) << 20) / job_scratch(cap))); }

template <class T>
T *take(char *&p, size_t n) {
    T *q = reinterpret_cast<T *>(p);
    p += (n * sizeof(T) + 255) / 256 * 256;
    return q;
}

Chains carve(void *scratch, int njobs, int cap) {
    char *p = static_cast<char *>(scratch);
    const size_t n = (size_t)njobs * 2 * cap;
    Chains ch;
    ch.parts = take<Part>(p, (size_t)njobs * cap);
    ch.pos = take<int64_t>(p, (size_t)njobs * 2 * (cap + 1));
    ch.start = take<int64_t>(p, n);
    ch.end = take<double>(p, n * kVar);
    ch.slack = take<double>(p, n * kVar);
    return ch;
}

template <class Job, int KIND0>
void launch_chain(const Job *d_jobs, int njobs, int nchains, const Chains &ch, int cap, int L, cudaStream_t s) {
    const int segs = kWarps * kSegs;
    const dim3 bounds((unsigned)((cap + 3) / 4), (unsigned)njobs, (unsigned)nchains);
    const dim3 sim((unsigned)((cap + segs - 1) / segs), (unsigned)njobs, (unsigned)nchains);
    const dim3 walk(1, (unsigned)njobs, (unsigned)nchains);
    bounds_kernel<Job, KIND0><<<bounds, 128, 0, s>>>(d_jobs, ch, cap, L);
    spec_kernel<Job, KIND0><<<sim, 32 * kWarps, 0, s>>>(d_jobs, ch, cap, L);
    if (KIND0 == kNyquist) {
        // Of 16-bit samples' alternating sums one segment in seven fails its
        // conditions and every fourth such prediction is wrong: all are
        // simulated again at once, from within a few ulps, instead of one
        // round of checks after the other (0.24 ms for 480,000 samples).
        resolve_kernel<Job, KIND0, true><<<walk, kBatch, 0, s>>>(d_jobs, ch, cap, L);
        spec_kernel<Job, KIND0><<<sim, 32 * kWarps, 0, s>>>(d_jobs, ch, cap, L);
        launch_counter() += 2;
    }
    resolve_kernel<Job, KIND0, false><<<walk, kBatch, 0, s>>>(d_jobs, ch, cap, L);
    launch_counter() += 3;
}

template <class Job>
void launch_parts(const Job *d_jobs, int njobs, const Chains &ch, int cap, int L, cudaStream_t s) {
    parts_kernel<Job><<<dim3((unsigned)((cap + 7) / 8), (unsigned)njobs), 256, 0, s>>>(d_jobs, ch.parts, cap, L);
    launch_counter() += 1;
}

}  // namespace

size_t serial_sum_scratch(int njobs, int64_t max_len) {
    const int cap = segment_cap(max_len);
    return (size_t)std::min(njobs, jobs_per_launch(cap)) * job_scratch(cap) + 5 * 256;
}

namespace {
template <class Job, class F>
void by_launches(const Job *d_jobs, int njobs, int64_t max_len, void *d_scratch, F &&f) {
    const int L = segment_length(max_len), cap = segment_cap(max_len), per = jobs_per_launch(cap);
    for (int i = 0; i < njobs; i += per) {
        const int n = std::min(per, njobs - i);
        f(d_jobs + i, n, carve(d_scratch, n, cap), cap, L);
    }
}
}  // namespace

void launch_envelope_stats(const SumJob *d_jobs, int njobs, int64_t max_len, void *d_scratch, cudaStream_t s) {
    by_launches(d_jobs, njobs, max_len, d_scratch, [&](const SumJob *j, int n, const Chains &ch, int cap, int L) {
        launch_parts(j, n, ch, cap, L, s);
        launch_chain<SumJob, kSum>(j, n, 2, ch, cap, L, s);
        launch_chain<SumJob, kNyquist>(j, n, 1, ch, cap, L, s);
    });
}

void launch_energy(const SumJob *d_jobs, int njobs, int64_t max_len, void *d_scratch, cudaStream_t s) {
    by_launches(d_jobs, njobs, max_len, d_scratch, [&](const SumJob *j, int n, const Chains &ch, int cap, int L) {
        launch_parts(j, n, ch, cap, L, s);
        launch_chain<SumJob, kEnergy>(j, n, 1, ch, cap, L, s);
    });
}

void launch_aligned_energy(const AlignedEnergyJob *d_jobs, int njobs, int64_t max_len, void *d_scratch, cudaStream_t s) {
    by_launches(d_jobs, njobs, max_len, d_scratch, [&](const AlignedEnergyJob *j, int n, const Chains &ch, int cap, int L) {
        launch_parts(j, n, ch, cap, L, s);
        launch_chain<AlignedEnergyJob, kEnergy>(j, n, 1, ch, cap, L, s);
    });
}

}  // namespace vqb
