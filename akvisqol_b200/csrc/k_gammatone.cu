// Gammatone filterbank spectrogram, exact form (reference
// src/gammatone.zig:268-306 and 432-467).
//
// Every (frame, band) RMS is an independent 4-biquad recurrence over one
// Hann-windowed frame from zero state, so one thread owns one (frame, band)
// and keeps the eight state values in registers. A CTA takes F consecutive
// frames of one job with all NB bands (thread = frame * NB + band) and stages
// their windowed samples, each product formed once, in shared memory 64 at a
// time; the next 64 are loaded into registers meanwhile.
//
// The work is FP64-pipe bound: 30 separately rounded f64 operations a sample
// (no FMA, as the CPU), 60 issue cycles of a warp's scheduler. The four
// biquads run skewed, stage k on sample i - k, so that a step holds four
// independent recurrences instead of one chain through all of them: the same
// operations on the same operands. That matters where a scheduler has one
// warp (a single pair's spectrogram is 500 warps on 592 schedulers): with the
// staging, 295 -> 173 us for 10 s at 48 kHz and 149 -> 65 us for 2.5 s of
// speech, against 122 and 41 us of pure issue.
#include <algorithm>

#include "device.cuh"
#include "kernels.h"

namespace vqb {

namespace {

struct Tile {
    int32_t job;
    int32_t frame0;
};

constexpr int kTileS = 64;        // samples staged at a time
constexpr int kRow = kTileS + 2;  // a frame's row of a stage (rows of a warp in different banks)

// Transposed direct form II with the CPU's operation order.
struct Biquad {
    double c0 = 0.0, c1 = 0.0;
    __device__ inline double step(double x, double n0, double n1, double d1, double d2) {
        const double y = n0 * x + c0;
        c0 = n1 * x + c1 - d1 * y;
        c1 = -(d2 * y);
        return y;
    }
};

// wx: [2][frames][kRow] windowed samples (dynamic shared memory).
__global__ void __launch_bounds__(256) gammatone_kernel(const SpecJob *__restrict__ jobs, const Tile *__restrict__ tiles,
                                                        const BandCoeffs *__restrict__ coeffs, int nb,
                                                        const double *__restrict__ hann, int window, int hop) {
    extern __shared__ __align__(16) double wx[];
    const Tile tile = tiles[blockIdx.x];
    const int frames = blockDim.x / nb;
    const int fl = threadIdx.x / nb;
    const int band = threadIdx.x - fl * nb;
    const SpecJob job = jobs[tile.job];
    const VSig sig = job.sig;
    const BandCoeffs k = coeffs[band];
    const int total = frames * kTileS;
    // entry e of a tile: frame e / kTileS, sample e % kTileS. A thread holds
    // its entries' samples of the next tile in registers (64 / nb of them, at
    // most kHold), the rest are loaded when they are windowed.
    constexpr int kHold = 4;
    double held[kHold];
    auto sample = [&](int e, int i0) {
        const int c = e / kTileS, i = i0 + (e - c * kTileS);
        return i < window ? vsig_at(sig, ((int64_t)tile.frame0 + c) * hop + i) : 0.0;
    };
    auto load = [&](int i0) {
#pragma unroll
        for (int m = 0; m < kHold; ++m) {
            const int e = threadIdx.x + m * blockDim.x;
            if (e < total) held[m] = sample(e, i0);
        }
    };
    auto store = [&](int i0, int buf) {
        double *w = wx + buf * frames * kRow;
        auto put = [&](int e, double x) {
            const int c = e / kTileS, j = e - c * kTileS, i = i0 + j;
            w[c * kRow + j] = i < window ? x * __ldg(hann + i) : 0.0;
        };
#pragma unroll
        for (int m = 0; m < kHold; ++m) {
            const int e = threadIdx.x + m * blockDim.x;
            if (e < total) put(e, held[m]);
        }
        for (int e = threadIdx.x + kHold * blockDim.x; e < total; e += blockDim.x) put(e, sample(e, i0));
    };
    Biquad s1, s2, s3, s4;
    double y1 = 0.0, y2 = 0.0, y3 = 0.0, sum_sq = 0.0;
    auto step = [&](double x) {
        const double y4 = s4.step(y3, k.ca0, k.s4n1, k.d1, k.d2);
        y3 = s3.step(y2, k.ca0, k.s3n1, k.d1, k.d2);
        y2 = s2.step(y1, k.ca0, k.s2n1, k.d1, k.d2);
        y1 = s1.step(x, k.s1n0, k.s1n1, k.d1, k.d2);
        sum_sq += y4 * y4;
    };
    load(0);
    store(0, 0);
    load(kTileS);
    __syncthreads();
    int buf = 0;
    for (int i0 = 0; i0 < window; i0 += kTileS, buf ^= 1) {
        const double *w = wx + (buf * frames + fl) * kRow;
        if (window - i0 >= kTileS) {
#pragma unroll 4
            for (int i = 0; i < kTileS; i += 2) {
                const double2 x = *reinterpret_cast<const double2 *>(w + i);
                step(x.x);
                step(x.y);
            }
        } else {
            for (int i = 0; i < window - i0; ++i) step(w[i]);
        }
        if (i0 + kTileS < window) {
            store(i0 + kTileS, buf ^ 1);
            if (i0 + 2 * kTileS < window) load(i0 + 2 * kTileS);
        }
        __syncthreads();
    }
    for (int i = 0; i < 3; ++i) step(0.0);  // the last three samples through the later stages
    const int64_t f = (int64_t)tile.frame0 + fl;
    if (f >= job.nf) return;
    const double inv_n = 1.0 / (double)window;
    job.out[(int64_t)band * job.nf + f] = sqrt(sum_sq * inv_n);
}

// The same recurrences for small launches: a CTA a frame, a warp eight bands,
// a band four lanes, one a biquad. Biquad q runs eight samples behind biquad
// q - 1, whose last outputs wait in shared memory. A lane's sample is seven
// operations with three in the chain (39 cycles) instead of 30; a warp issues
// 18 cycles a sample for eight (frame, band)s instead of 62 for 32.
constexpr int kSub = 8;
constexpr int kBlock = 64;  // samples staged at a time, by each warp for itself
struct __align__(16) SplitShared {
    double x[kBlock];
    double box[2][32][kSub + 2];  // by parity of the step (16-byte accesses of eight lanes on distinct banks)
};

__global__ void __launch_bounds__(256) gammatone_split_kernel(const SpecJob *__restrict__ jobs,
                                                              const Tile *__restrict__ tiles,
                                                              const BandCoeffs *__restrict__ coeffs, int nb,
                                                              const double *__restrict__ hann, int window, int hop) {
    extern __shared__ __align__(16) double split_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = lane & 3;
    SplitShared &sm = reinterpret_cast<SplitShared *>(split_raw)[warp];
    const Tile tile = tiles[blockIdx.x];
    const SpecJob job = jobs[tile.job];
    const int raw = warp * 8 + (lane >> 2), band = min(raw, nb - 1);
    const BandCoeffs k = coeffs[band];
    const double n0 = q == 0 ? k.s1n0 : k.ca0, n1 = q == 0 ? k.s1n1 : q == 1 ? k.s2n1 : q == 2 ? k.s3n1 : k.s4n1;
    const double d1 = k.d1, d2 = k.d2;
    const int64_t k0 = (int64_t)tile.frame0 * hop;
    double px[kBlock / 32], ph[kBlock / 32];
    auto load = [&](int i0) {
#pragma unroll
        for (int m = 0; m < kBlock / 32; ++m) {
            const int i = i0 + 32 * m + lane;
            px[m] = i < window ? vsig_at(job.sig, k0 + i) : 0.0;
            ph[m] = i < window ? __ldg(hann + i) : 0.0;
        }
    };
#pragma unroll
    for (int j = 0; j < kSub; ++j) sm.box[0][lane][j] = sm.box[1][lane][j] = 0.0;
    double c0 = 0.0, c1 = 0.0, sum = 0.0, v[kSub] = {};
    int par = 0;
    // eight samples of every biquad; biquad 4's outputs of the step before are
    // squared and added meanwhile (`left` of them lie inside the window)
    auto step = [&](const double *first, int left) {
        const double *in = q ? sm.box[par][lane - 1] : first;
        double x[kSub];
#pragma unroll
        for (int j = 0; j < kSub; j += 2) {
            const double2 t = *reinterpret_cast<const double2 *>(in + j);
            x[j] = t.x, x[j + 1] = t.y;
        }
#pragma unroll
        for (int j = 0; j < kSub; ++j) {
            const double z = j < left ? v[j] : 0.0;
            sum += z * z;
            const double y = n0 * x[j] + c0;
            c0 = n1 * x[j] + c1 - d1 * y;
            c1 = -(d2 * y);
            v[j] = y;
        }
        par ^= 1;
#pragma unroll
        for (int j = 0; j < kSub; j += 2)
            *reinterpret_cast<double2 *>(&sm.box[par][lane][j]) = make_double2(v[j], v[j + 1]);
        __syncwarp();
    };
    load(0);
    int i = 0;
    for (; i < window; i += kBlock) {
        __syncwarp();
#pragma unroll
        for (int m = 0; m < kBlock / 32; ++m) sm.x[32 * m + lane] = px[m] * ph[m];
        __syncwarp();
        load(i + kBlock);
        for (int s = 0; s < kBlock; s += kSub) step(sm.x + s, window - (i + s - 4 * kSub));
    }
    for (int s = 0; s < 4 * kSub; s += kSub) step(sm.x, window - (i + s - 4 * kSub));  // the rest through the later biquads
    if (q != 3 || raw >= nb) return;
    job.out[(int64_t)band * job.nf + tile.frame0] = sqrt(sum * (1.0 / (double)window));
}

// Grid-aligned frames copied from a full-signal spectrogram (reference
// src/realign.zig:262-281): dst[b*ncols + c] = src[b*stride + col + c].
__global__ void __launch_bounds__(256) copy_frames_kernel(const CopyJob *__restrict__ jobs, int nb) {
    const CopyJob job = jobs[blockIdx.y];
    const int total = nb * job.ncols;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const int b = e / job.ncols, c = e - b * job.ncols;
        job.dst[e] = job.src[(int64_t)b * job.src_stride + job.src_col + c];
    }
}

}  // namespace

// 128 threads: one warp a scheduler, and a few CTAs an SM in a large launch.
// Measured against 256, 64 and 32 threads (spectrogram kernels of a pass, us):
// one 10 s 48 kHz pair 519 (844, 518, 552), one 2.5 s speech pair 130 (204,
// 133, 153), 32 10 s pairs level.
//
// Launches of up to two warps a scheduler in the split form take it: 122
// speech frames 36 us (65 with a thread a band), 111 audio frames 103 (175),
// 262 audio frames 122 (170). At 497 audio frames, 3.4 warps a scheduler, its
// nine operations a lane, where a thread's share is 7.5, take 230 (173).
int gammatone_frames_per_cta(int nb, int64_t frames) {
    if (frames * ((nb + 7) / 8) <= 2 * 4 * 148) return kGammatoneSplit;
    return std::max(1, std::min(128 / nb, 16));
}

std::vector<int> gammatone_frames_shapes(int nb) {
    const int f = std::max(1, std::min(128 / nb, 16));
    std::vector<int> c{f, 2 * f};
    if (f / 2 >= 1) c.push_back(f / 2);
    return c;
}
size_t gammatone_tile_size() { return sizeof(Tile); }
void fill_gammatone_tile(void *dst, int job, int frame0) { *static_cast<Tile *>(dst) = Tile{job, frame0}; }

void launch_gammatone(const SpecJob *d_jobs, const void *d_tiles, int ntiles, const BandCoeffs *d_coeffs, int nb,
                      const double *d_hann, int window, int hop, int frames_per_cta, cudaStream_t s) {
    if (ntiles <= 0) return;
    launch_counter() += 1;
    if (frames_per_cta == kGammatoneSplit) {
        const int warps = (nb + 7) / 8;
        gammatone_split_kernel<<<ntiles, warps * 32, warps * sizeof(SplitShared), s>>>(
            d_jobs, static_cast<const Tile *>(d_tiles), d_coeffs, nb, d_hann, window, hop);
        return;
    }
    const int threads = frames_per_cta * nb;
    const size_t smem = (size_t)2 * frames_per_cta * kRow * sizeof(double);
    gammatone_kernel<<<ntiles, threads, smem, s>>>(d_jobs, static_cast<const Tile *>(d_tiles), d_coeffs, nb, d_hann,
                                               window, hop);
}

void launch_copy_frames(const CopyJob *d_jobs, int njobs, int nb, int max_cols, cudaStream_t s) {
    if (njobs <= 0) return;
    const int total = nb * max_cols;
    const int blocks = (total + 255) / 256;
    copy_frames_kernel<<<dim3((unsigned)(blocks < 1 ? 1 : blocks), (unsigned)njobs), 256, 0, s>>>(d_jobs, nb);
    launch_counter() += 1;
}

}  // namespace vqb
