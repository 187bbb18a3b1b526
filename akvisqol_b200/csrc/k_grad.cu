// Reverse of the gammatone RMS spectrogram (reference src/gpu/pipeline.zig:842-1143,
// its gammatone_bwd kernel): from d loss / d RMS cell to d loss / d sample.
//
// One (frame, band) is RMS = post sqrt(sum_i y_i^2 / W) with y the unit
// cascade of four biquads (direct form I, numerators 1 + beta z^-1, the
// FP64-FMA form's arithmetic) over the Hann-windowed frame x_i. So
//
//   d loss / d x = H^T (g post^2 / (W RMS) y),
//
// H the cascade as a lower-triangular Toeplitz map over the frame (zero
// state at its start). H^T is H run backwards in time (zero state at the
// frame's end): reverse the sequence, filter with the same four stages,
// reverse again. The sequence it filters is y in reverse order, so y is
// recomputed block by block, last block first, from states the forward
// pass saves every kBlock samples (in global scratch).
//
// A CTA is a frame, a warp eight of its bands, and a band four lanes, one a
// stage: stage q runs a sub-block of eight samples behind stage q - 1, whose
// outputs wait in shared memory (16-byte accesses), so a sample is three FP64
// instructions in one dependent chain instead of 13 in four. Stage 3's
// outputs are summed over the warp's bands 32 samples at a time, a lane a
// sample, and added to the samples' gradient by atomics (four frames overlap
// a sample, four warps hold its bands). Bound by the chains' latency: a pair
// has a warp for every other scheduler. A lane that ran all four stages of
// a band, and summed each sample over 32 lanes, took 1.86 ms for a 2.4 s
// 48 kHz pair, this takes 0.30; with shuffles between the stages and for
// the sums, four times the instructions, it took 0.56.
#include "device.cuh"
#include "kernels.h"

namespace vqb {

namespace {

constexpr int kSub = 8;           // samples of a sub-block
constexpr int kSubs = 16;         // sub-blocks of a block
constexpr int kBlock = kSub * kSubs;  // samples between saved states
constexpr int kState = 3;         // doubles of a stage's state
constexpr int kMaxWarps = 4;
// (rows padded so that 16-byte accesses of eight lanes fall on distinct banks)
constexpr int kRow = kBlock + 2;
constexpr int kBox = kSub + 2;
constexpr int kOut = 32 + 2;

struct __align__(16) WarpShared {
    double x[kBlock];         // a block's windowed samples
    double box[2][32][kBox];  // each lane's last sub-block of outputs, by parity of the step
    double y[8][kRow];        // a block's scaled y of each band, last sample first
    double out[8][kOut];      // each band's d loss / d sample, 32 samples
};

// One stage of the cascade: y = v + beta v[-1] - d2 y[-2] - d1 y[-1].
struct Stage {
    double v1 = 0.0, y1 = 0.0, y2 = 0.0;
    __device__ inline void run(double (&v)[kSub], double beta, double nd1, double nd2) {
#pragma unroll
        for (int j = 0; j < kSub; ++j) {
            const double y = __fma_rn(nd1, y1, __fma_rn(nd2, y2, __fma_rn(beta, v1, v[j])));
            v1 = v[j];
            y2 = y1;
            y1 = y;
            v[j] = y;
        }
    }
};

__device__ inline void get(double (&v)[kSub], const double *p) {
#pragma unroll
    for (int j = 0; j < kSub; j += 2) {
        const double2 t = *reinterpret_cast<const double2 *>(p + j);
        v[j] = t.x, v[j + 1] = t.y;
    }
}
__device__ inline void put(const double (&v)[kSub], double *p) {
#pragma unroll
    for (int j = 0; j < kSub; j += 2) *reinterpret_cast<double2 *>(p + j) = make_double2(v[j], v[j + 1]);
}

struct GradTile {
    int32_t job, frame0;
};

// grid: tiles of one frame; block: a warp per eight bands. scratch: per block
// and thread nblk x kState.
__global__ void __launch_bounds__(kMaxWarps * 32) gammatone_bwd_kernel(const GradSpecJob *__restrict__ jobs,
                                                                       const GradTile *__restrict__ tiles,
                                                                       const FastBandCoeffs *__restrict__ coeffs, int nb,
                                                                       const double *__restrict__ hann, int window,
                                                                       int hop, double *__restrict__ scratch) {
    extern __shared__ __align__(16) char sm_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = lane & 3, slot = lane >> 2;
    WarpShared &sm = reinterpret_cast<WarpShared *>(sm_raw)[warp];
    const GradTile tile = tiles[blockIdx.x];
    const GradSpecJob job = jobs[tile.job];
    const int64_t f = tile.frame0;
    const int raw = warp * 8 + slot, band = min(raw, nb - 1);
    const double g = raw < nb ? job.g_rms[(int64_t)band * job.nf + f] : 0.0;
    if (!__any_sync(0xffffffffu, g != 0.0)) return;  // warp-uniform: no gradient in these bands
    const FastBandCoeffs k = coeffs[band];
    const double beta = k.beta64[q], nd1 = -k.d1, nd2 = -k.d2;
    const int nblk = (window + kBlock - 1) / kBlock;
    double *ck = scratch + ((int64_t)blockIdx.x * nblk * kState) * blockDim.x + threadIdx.x;
    const int64_t k0 = f * hop;

    // a block's windowed samples, zero behind the window: read a block ahead,
    // then into the warp's shared memory
    double px[kBlock / 32], ph[kBlock / 32];
    auto fetch = [&](int blk) {
#pragma unroll
        for (int m = 0; m < kBlock / 32; ++m) {
            const int i = blk * kBlock + 32 * m + lane;
            const bool in = blk >= 0 && i < window;
            px[m] = in ? vsig_at(job.sig, k0 + i) : 0.0;
            ph[m] = in ? __ldg(hann + i) : 0.0;
        }
    };
    auto stage_x = [&] {
        __syncwarp();
#pragma unroll
        for (int m = 0; m < kBlock / 32; ++m) sm.x[32 * m + lane] = px[m] * ph[m];
        __syncwarp();
    };
    // a step of every stage: stage 0's inputs from `first`, the others' from
    // the lane before (what it left in the step before)
    int par = 0;
    auto clear = [&] {
        __syncwarp();
#pragma unroll
        for (int j = 0; j < kSub; ++j) sm.box[0][lane][j] = sm.box[1][lane][j] = 0.0;
        __syncwarp();
    };
    auto step = [&](Stage &st, double (&v)[kSub], const double *first) {
        get(v, q ? sm.box[par][lane - 1] : first);
        st.run(v, beta, nd1, nd2);
        par ^= 1;
        put(v, sm.box[par][lane]);
        __syncwarp();
    };

    // forward: sum of squares of y, each stage's state at each block's start
    // (stages behind the first run on zeros until the first sub-block reaches them)
    Stage st;
    double v[kSub], ss = 0.0;
    auto square = [&](int i) {  // stage 3's sub-block at sample i (the other stages' sums are not used)
        double a = 0.0, b = 0.0;
        if (i + kSub > window) {
#pragma unroll
            for (int j = 0; j < kSub; ++j) v[j] = i + j < window ? v[j] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < kSub; j += 2) a = __fma_rn(v[j], v[j], a), b = __fma_rn(v[j + 1], v[j + 1], b);
        ss += a + b;
    };
    clear();
    fetch(0);
    for (int blk = 0; blk < nblk; ++blk) {
        stage_x();
        fetch(blk + 1 < nblk ? blk + 1 : -1);
        for (int s = 0; s < kSubs; ++s) {
            if (s == q) {
                double *p = ck + (int64_t)blk * kState * blockDim.x;
                p[0] = st.v1, p[blockDim.x] = st.y1, p[2 * blockDim.x] = st.y2;
            }
            step(st, v, sm.x + s * kSub);
            square((blk * kSubs + s - 3) * kSub);
        }
    }
    for (int s = 0; s < 3; ++s) {  // the last sub-blocks reach stage 3
        step(st, v, sm.x);
        square((nblk * kSubs + s - 3) * kSub);
    }
    ss = __shfl_sync(0xffffffffu, ss, 3, 4);
    const double rms = sqrt(ss / (double)window) * k.post64;
    // d loss / d y_i = scale y_i
    const double scale = rms > 0.0 ? g * k.post64 * k.post64 / ((double)window * rms) : 0.0;

    // reverse: blocks last to first; a block's y recomputed, then fed
    // backwards through the same cascade
    Stage back;
    double held[kSub] = {};  // the reverse pass's outputs while the boxes serve a recomputation
    const int top = nblk * kBlock - 1;
    auto add = [&](int u) {  // reverse sub-block u (samples top - 8 u - j) has left stage 3
        if (u < 0) return;
        if (q == 3) put(held, sm.out[slot] + u % 4 * kSub);
        if (u % 4 != 3) return;
        __syncwarp();
        double a = sm.out[0][lane], b = sm.out[1][lane];
#pragma unroll
        for (int m = 2; m < 8; m += 2) a += sm.out[m][lane], b += sm.out[m + 1][lane];
        __syncwarp();
        const int i = top - kSub * (u - 3) - lane;
        const int64_t at = k0 + i - job.sig.head;
        if (i < window && (uint64_t)at < (uint64_t)job.sig.avail) atomicAdd(job.grad + at, (a + b) * __ldg(hann + i));
    };
    fetch(nblk - 1);
    for (int blk = nblk - 1; blk >= 0; --blk) {
        stage_x();
        fetch(blk - 1);
        Stage saved;
        {
            const double *p = ck + (int64_t)blk * kState * blockDim.x;
            saved.v1 = p[0], saved.y1 = p[blockDim.x], saved.y2 = p[2 * blockDim.x];
        }
        for (int s = 0; s < kSubs + 3; ++s) {  // (a stage's steps before its first sub-block and behind its last go nowhere)
            if (s == q) st = saved;
            step(st, v, sm.x + (s < kSubs ? s : 0) * kSub);
            if (q == 3 && s >= 3) {
                const int i = (s - 3) * kSub;
                double z[kSub];
#pragma unroll
                for (int j = 0; j < kSub; ++j) z[j] = blk * kBlock + i + kSub - 1 - j < window ? scale * v[kSub - 1 - j] : 0.0;
                put(z, sm.y[slot] + kBlock - kSub - i);
            }
        }
        // the reverse pass's last outputs back into the boxes
        put(held, sm.box[par][lane]);
        __syncwarp();
        const int u0 = (nblk - 1 - blk) * kSubs;
        for (int s = 0; s < kSubs; ++s) {
            step(back, held, sm.y[slot] + s * kSub);
            add(u0 + s - 3);
        }
    }
    for (int s = 0; s < 3; ++s) {
        step(back, held, sm.x);
        add(nblk * kSubs + s - 3);
    }
}

}  // namespace

size_t gammatone_bwd_scratch_count(int ntiles, int window) {
    return (size_t)ntiles * kMaxWarps * 32 * (size_t)((window + kBlock - 1) / kBlock) * kState;
}

void launch_gammatone_bwd(const GradSpecJob *d_jobs, const void *d_tiles, int ntiles, const FastBandCoeffs *d_coeffs,
                          int nb, const double *d_hann, int window, int hop, double *d_scratch, cudaStream_t s) {
    if (ntiles <= 0) return;
    cudaFuncSetAttribute(gammatone_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         kMaxWarps * (int)sizeof(WarpShared));
    const int warps = (nb + 7) / 8;
    gammatone_bwd_kernel<<<ntiles, warps * 32, warps * sizeof(WarpShared), s>>>(
        d_jobs, static_cast<const GradTile *>(d_tiles), d_coeffs, nb, d_hann, window, hop, d_scratch);
    launch_counter() += 1;
}

}  // namespace vqb
