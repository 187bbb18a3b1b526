// Signal-level kernels: the FMA forms' statistics as tree sums, upper
// envelopes packed for the lag FFT, and the lag/SPL application (the exact
// form's sums in the CPU's order are in k_sums.cu).
#include "device.cuh"
#include "kernels.h"

namespace vqb {

namespace {

// ---- fast form: tree reductions -------------------------------------------
// The fast form does not reproduce the CPU's rounding, so its statistics are
// deterministic tree sums: kTreeParts CTAs per signal each reduce a
// contiguous range (strided, coalesced loads; warp shuffles; shared memory)
// into scratch, and one warp per signal adds the parts in order.
constexpr int kTreeThreads = 256;

__device__ inline double block_sum(double v, double *sm) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sm[wid] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x < 32) {
        t = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    }
    return t;  // valid in thread 0
}

__device__ inline void part_range(int64_t n, int64_t &lo, int64_t &hi) {
    const int64_t per = (n + kTreeParts - 1) / kTreeParts;
    lo = per * blockIdx.x;
    hi = lo + per < n ? lo + per : n;
}

// Partial sums of x, (-1)^k x and x^2 over this CTA's range.
__global__ void __launch_bounds__(kTreeThreads) stats_tree_parts(const SumJob *__restrict__ jobs,
                                                                 double *__restrict__ scratch) {
    __shared__ double sm[kTreeThreads / 32];
    const SumJob job = jobs[blockIdx.y];
    int64_t lo, hi;
    part_range(job.sig.len, lo, hi);
    double s = 0.0, a = 0.0, e = 0.0;
#pragma unroll 4
    for (int64_t k = lo + threadIdx.x; k < hi; k += kTreeThreads) {
        const double x = vsig_at(job.sig, k);
        s += x;
        a += (k & 1) ? -x : x;
        e = __fma_rn(x, x, e);
    }
    s = block_sum(s, sm);
    a = block_sum(a, sm);
    e = block_sum(e, sm);
    if (threadIdx.x == 0) {
        double *p = scratch + ((int64_t)blockIdx.y * kTreeParts + blockIdx.x) * 3;
        p[0] = s;
        p[1] = a;
        p[2] = e;
    }
}

// out[0] = sum x, out[1] = sum (-1)^k (x - mean) = alt - mean * (len odd),
// out[2] = sum x^2.
__global__ void __launch_bounds__(32) stats_tree_finish(const SumJob *__restrict__ jobs,
                                                        const double *__restrict__ scratch) {
    const SumJob job = jobs[blockIdx.x];
    const double *p = scratch + (int64_t)blockIdx.x * kTreeParts * 3;
    const int lane = threadIdx.x;
    double s = p[lane * 3], a = p[lane * 3 + 1], e = p[lane * 3 + 2];
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, o);
        a += __shfl_down_sync(0xffffffffu, a, o);
        e += __shfl_down_sync(0xffffffffu, e, o);
    }
    if (lane == 0) {
        const int64_t len = job.sig.len;
        const double mean = len > 0 ? s / (double)len : 0.0;
        job.out[0] = s;
        job.out[1] = (len & 1) ? a - mean : a;
        job.out[2] = e;
    }
}

// Aligned energy as a tree sum.
__global__ void __launch_bounds__(kTreeThreads) aligned_tree_parts(const AlignedEnergyJob *__restrict__ jobs,
                                                                   double *__restrict__ scratch) {
    __shared__ double sm[kTreeThreads / 32];
    const AlignedEnergyJob job = jobs[blockIdx.y];
    int64_t skip, alen;
    aligned_range(job, skip, alen);
    int64_t lo, hi;
    part_range(job.deg.len - skip, lo, hi);
    double e = 0.0;
#pragma unroll 4
    for (int64_t k = lo + threadIdx.x; k < hi; k += kTreeThreads) {
        const double x = vsig_at(job.deg, skip + k);
        e = __fma_rn(x, x, e);
    }
    e = block_sum(e, sm);
    if (threadIdx.x == 0) scratch[((int64_t)blockIdx.y * kTreeParts + blockIdx.x) * 3] = e;
}

__global__ void __launch_bounds__(32) aligned_tree_finish(const AlignedEnergyJob *__restrict__ jobs,
                                                          const double *__restrict__ scratch) {
    const AlignedEnergyJob job = jobs[blockIdx.x];
    double e = scratch[((int64_t)blockIdx.x * kTreeParts + threadIdx.x) * 3];
    for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
    if (threadIdx.x == 0) {
        int64_t skip, alen;
        aligned_range(job, skip, alen);
        job.out[0] = e;
        job.out[1] = (double)alen;
    }
}

__host__ __device__ inline int64_t next_pow_two(int64_t x) {
    int64_t n = 1;
    while (n < x) n <<= 1;
    return n;
}

// upperEnvelope's closed form (reference src/envelope.zig:23-53) for both
// signals of a lag job, packed as z = env_a + i env_b zero-padded to n
// (reference src/xcorr.zig:204-208). raw: the signals themselves.
template <bool RAW>
__global__ void __launch_bounds__(256) pack_kernel(const LagJob *__restrict__ jobs, int njobs) {
    const LagJob job = jobs[blockIdx.y];
    const int64_t n = job.n;
    double mean_a = 0, q_a = 0, mean_b = 0, q_b = 0;
    if (!RAW) {
        const int64_t la = job.a.len, lb = job.b.len;
        if (la > 0) {
            mean_a = job.stats_a[0] / (double)la;
            const int64_t Na = next_pow_two(la) > 32 ? next_pow_two(la) : 32;
            q_a = job.stats_a[1] / (double)Na;
        }
        if (lb > 0) {
            mean_b = job.stats_b[0] / (double)lb;
            const int64_t Nb = next_pow_two(lb) > 32 ? next_pow_two(lb) : 32;
            q_b = job.stats_b[1] / (double)Nb;
        }
    }
    const double eps = 0.000001;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double re = 0.0, im = 0.0;
        if (i < job.a.len) {
            const double x = vsig_at(job.a, i);
            if (RAW) {
                re = x;
            } else {
                const double pc = x - mean_a;
                const double nt = (i & 1) ? -q_a : q_a;
                re = fabs(2.0 * (pc - nt) - eps) + mean_a;
            }
        }
        if (i < job.b.len) {
            const double x = vsig_at(job.b, i);
            if (RAW) {
                im = x;
            } else {
                const double pc = x - mean_b;
                const double nt = (i & 1) ? -q_b : q_b;
                im = fabs(2.0 * (pc - nt) - eps) + mean_b;
            }
        }
        job.z[i] = make_double2(re, im);
    }
}

// ---- speech VAD -------------------------------------------------------------
// The samples scale to the signal's peak and truncate to int16, so a chunk's
// sum of squares is an integer far below 2^53: any order gives the CPU's sum.

// Partial maxima (NaN samples left out, as the CPU's @max).
__global__ void __launch_bounds__(kTreeThreads) vad_peak_kernel(const VadJob *__restrict__ jobs,
                                                                double *__restrict__ scratch) {
    __shared__ double sm[kTreeThreads / 32];
    const VadJob job = jobs[blockIdx.y];
    int64_t lo, hi;
    part_range(job.sig.len, lo, hi);
    double m = -INFINITY;
#pragma unroll 4
    for (int64_t k = lo + threadIdx.x; k < hi; k += kTreeThreads) m = fmax(m, vsig_at(job.sig, k));
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kTreeThreads / 32; ++w) m = fmax(m, sm[w]);
        scratch[(int64_t)blockIdx.y * kTreeParts + blockIdx.x] = m;
    }
}

// A warp per chunk.
__global__ void __launch_bounds__(128) vad_loud_kernel(const VadJob *__restrict__ jobs,
                                                       const double *__restrict__ scratch) {
    const VadJob job = jobs[blockIdx.y];
    const int lane = threadIdx.x & 31, c = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (c >= job.chunks) return;
    double peak = scratch[(int64_t)blockIdx.y * kTreeParts + lane];
    for (int o = 16; o > 0; o >>= 1) peak = fmax(peak, __shfl_xor_sync(0xffffffffu, peak, o));
    const int64_t k0 = job.first + (int64_t)c * job.frame_len;
    double sq = 0.0;
    for (int j = lane; j < job.frame_len; j += 32) {
        const int64_t k = k0 + j;
        const double v = (k < job.sig.len ? vsig_at(job.sig, k) / peak : 0.0) * 32768.0;
        const double s = trunc(v < -32768.0 ? -32768.0 : v > 32767.0 ? 32767.0 : v);  // (NaN stays)
        sq += s * s;
    }
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (lane == 0) job.loud[c] = sqrt(sq / (double)job.frame_len) >= 5000.0 ? 1 : 0;
}

// out[i] = aligned(i) * factor: scaleToMatchSpl on the lag-aligned signal
// (reference src/audio.zig:152-158; x * 1.0 == x when unscaled).
struct ScaleArgs {
    VSig src;
    double factor;
    double *out;
};

__global__ void __launch_bounds__(256) scale_kernel(const ScaleArgs *__restrict__ jobs, int njobs) {
    const ScaleArgs job = jobs[blockIdx.y];
#pragma unroll 4
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < job.src.len;
         i += (int64_t)gridDim.x * blockDim.x)
        job.out[i] = vsig_at(job.src, i) * job.factor;
}

}  // namespace

uint64_t &launch_counter() {
    static thread_local uint64_t count = 0;
    return count;
}

void launch_envelope_stats_tree(const SumJob *d_jobs, int njobs, double *d_scratch, cudaStream_t s) {
    if (njobs <= 0) return;
    static_assert(kTreeParts == 32, "the finishing warp adds one part per lane");
    stats_tree_parts<<<dim3(kTreeParts, (unsigned)njobs), kTreeThreads, 0, s>>>(d_jobs, d_scratch);
    stats_tree_finish<<<njobs, 32, 0, s>>>(d_jobs, d_scratch);
    launch_counter() += 2;
}

void launch_aligned_energy_tree(const AlignedEnergyJob *a, int njobs, double *d_scratch, cudaStream_t s) {
    if (njobs <= 0) return;
    aligned_tree_parts<<<dim3(kTreeParts, (unsigned)njobs), kTreeThreads, 0, s>>>(a, d_scratch);
    aligned_tree_finish<<<njobs, 32, 0, s>>>(a, d_scratch);
    launch_counter() += 2;
}

void launch_vad(const VadJob *d_jobs, int njobs, int max_chunks, double *d_scratch, cudaStream_t s) {
    if (njobs <= 0 || max_chunks <= 0) return;
    vad_peak_kernel<<<dim3(kTreeParts, (unsigned)njobs), kTreeThreads, 0, s>>>(d_jobs, d_scratch);
    vad_loud_kernel<<<dim3((unsigned)((max_chunks + 3) / 4), (unsigned)njobs), 128, 0, s>>>(d_jobs, d_scratch);
    launch_counter() += 2;
}

void launch_pack(const LagJob *d_jobs, int njobs, int64_t max_n, bool raw, cudaStream_t s) {
    if (njobs <= 0) return;
    const int threads = 256;
    int64_t blocks = (max_n + threads - 1) / threads;
    if (blocks > 4096) blocks = 4096;
    dim3 grid((unsigned)blocks, (unsigned)njobs);
    if (raw)
        pack_kernel<true><<<grid, threads, 0, s>>>(d_jobs, njobs);
    else
        pack_kernel<false><<<grid, threads, 0, s>>>(d_jobs, njobs);
    launch_counter() += 1;
}

size_t scale_args_size() { return sizeof(ScaleArgs); }
void fill_scale_args(void *dst, const VSig &src, double factor, double *out) {
    *static_cast<ScaleArgs *>(dst) = ScaleArgs{src, factor, out};
}
void launch_scale(const void *d_args, int njobs, int64_t max_len, cudaStream_t s) {
    if (njobs <= 0) return;
    // eight or more samples a thread: a CTA per 2048 samples, at most 256 a
    // signal (one sample a thread made block scheduling the cost)
    const int threads = 256;
    int64_t blocks = (max_len + 8 * threads - 1) / (8 * threads);
    if (blocks > 256) blocks = 256;
    if (blocks < 1) blocks = 1;
    scale_kernel<<<dim3((unsigned)blocks, (unsigned)njobs), threads, 0, s>>>(static_cast<const ScaleArgs *>(d_args),
                                                                            njobs);
    launch_counter() += 1;
}

}  // namespace vqb
