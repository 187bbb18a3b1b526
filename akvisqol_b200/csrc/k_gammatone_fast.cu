// Gammatone filterbank spectrograms of the FMA forms by the recurrence itself:
// the cascade of four biquads per (frame, band) of the exact kernel (reference
// src/gammatone.zig:268-306) without its operation order. It serves the
// windows that the spectral kernels (k_spectral.cu) do not: sample rates above
// 51.2 kHz or up to 6.4 kHz.
//
// Each biquad runs in direct form I with its numerator normalised to
// 1 + beta z^-1 (the four numerator gains and the band gain become one
// factor on the RMS), so a stage is three FMAs: y = v + beta v[-1] - d2 y[-2]
// - d1 y[-1], 13 FMAs and one multiply per sample instead of the exact form's
// 31 separately rounded operations.
//
// The CTA's 16 frames are Hann-windowed once per 64-sample tile into shared
// memory (double-buffered; the next tile's samples arrive by asynchronous
// copies while the current one is filtered), so a thread reads its two
// frames' windowed samples with one 16-byte load per step. A warp holds 8
// bands x 4 frame pairs: lanes of a frame pair read the same shared-memory
// word (a broadcast). A CTA holds ceil(nb/8) band groups x 2 frame blocks of
// 8 frames. Bound by the FP64 pipe: 0.82 of its measured FMA peak over a
// large batch.
#include <algorithm>

#include "device.cuh"
#include "kernels.h"

namespace vqb {

namespace {

struct Tile {
    int32_t job;
    int32_t frame0;
};

constexpr int kFramesPerBlock = 8;   // frames per warp (4 lanes rows x 2)
constexpr int kBlocksPerCta = 2;
constexpr int kCtaFrames = kFramesPerBlock * kBlocksPerCta;
constexpr int kTileS = 64;           // samples per shared-memory tile
constexpr int kRowPad = kCtaFrames + 2;  // doubles per tile row (2-way write conflicts, 16-byte reads)

// 8-byte asynchronous global-to-shared copy; bytes = 0 writes zeros.
__device__ inline void cp_async8(double *dst, const double *src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ inline void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ inline void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// The four stages of one frame and its sum of squares. Two frames run per
// thread (the second hop samples later): two independent recurrences give each
// warp twice the FP64 work between dependent steps.
struct Cascade64 {
    double xp = 0.0, y1a = 0.0, y2a = 0.0, y1b = 0.0, y2b = 0.0, y1c = 0.0, y2c = 0.0, y1d = 0.0, y2d = 0.0;
    double acc = 0.0;
    __device__ inline void step(double x, double b0, double b1, double b2, double b3, double nd1, double nd2) {
        // stage k input v, previous input = stage k-1's previous output
        const double ya = __fma_rn(nd1, y1a, __fma_rn(nd2, y2a, __fma_rn(b0, xp, x)));
        const double yb = __fma_rn(nd1, y1b, __fma_rn(nd2, y2b, __fma_rn(b1, y1a, ya)));
        const double yc = __fma_rn(nd1, y1c, __fma_rn(nd2, y2c, __fma_rn(b2, y1b, yb)));
        const double yd = __fma_rn(nd1, y1d, __fma_rn(nd2, y2d, __fma_rn(b3, y1c, yc)));
        xp = x;
        y2a = y1a;
        y1a = ya;
        y2b = y1b;
        y1b = yb;
        y2c = y1c;
        y1c = yc;
        y2d = y1d;
        y1d = yd;
        acc = __fma_rn(yd, yd, acc);
    }
};

// One staged tile through both of a thread's cascades.
__device__ inline void filter_tile(const double (*__restrict__ wx)[kRowPad], int q, int count,
                                     const FastBandCoeffs &k, Cascade64 &A, Cascade64 &B) {
    const double b0 = k.beta64[0], b1 = k.beta64[1], b2 = k.beta64[2], b3 = k.beta64[3];
    const double nd1 = -k.d1, nd2 = -k.d2;
    auto step = [&](int i) {
        const double2 w = *reinterpret_cast<const double2 *>(&wx[i][q]);
        A.step(w.x, b0, b1, b2, b3, nd1, nd2);
        B.step(w.y, b0, b1, b2, b3, nd1, nd2);
    };
    if (count == kTileS) {
#pragma unroll 4
        for (int i = 0; i < kTileS; ++i) step(i);
    } else {
        for (int i = 0; i < count; ++i) step(i);
    }
}

// One tile (16 frames x all bands of one job) a CTA. raw: signal samples,
// frame-major; wx: windowed samples, sample-major. kThreads = 64 x ceil(nb / 8):
// 256 for 32 bands, 192 for 21; two CTAs an SM (110 registers).
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 2 * 256 / kThreads) gammatone_staged_kernel(
    const SpecJob *__restrict__ jobs, const Tile *__restrict__ tiles, const FastBandCoeffs *__restrict__ coeffs, int nb,
    const double *__restrict__ hann, int window, int hop) {
    __shared__ __align__(16) double raw[2][kCtaFrames][kTileS];
    __shared__ __align__(16) double wx[2][kTileS][kRowPad];
    const Tile tile = tiles[blockIdx.x];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int groups = (nb + 7) >> 3;
    const int g = warp % groups, fblock = warp / groups;
    const int band_raw = g * 8 + (lane & 7);
    const int band = band_raw < nb ? band_raw : nb - 1;  // idle lanes filter a real band, never write
    const int q = fblock * kFramesPerBlock + 2 * (lane >> 3);
    const SpecJob job = jobs[tile.job];
    const VSig sig = job.sig;
    const int64_t f = (int64_t)tile.frame0 + q;
    const FastBandCoeffs k = coeffs[band];

    // Tiles of kTileS samples of the CTA's frames: entry e = (frame c =
    // e / kTileS, sample i = e % kTileS), so consecutive threads copy
    // consecutive samples of a frame. Samples outside the signal's stored
    // range or past the window are zero-filled by the copy itself.
    constexpr int kFills = (kCtaFrames * kTileS + kThreads - 1) / kThreads;
    auto fetch = [&](int i0, int buf) {
#pragma unroll
        for (int m = 0; m < kFills; ++m) {
            const int e = threadIdx.x + m * kThreads;
            if (e < kCtaFrames * kTileS) {
                const int c = e / kTileS, i = e - c * kTileS;
                const int64_t j = ((int64_t)tile.frame0 + c) * hop + i0 + i - sig.head;
                const bool in = i0 + i < window && (uint64_t)j < (uint64_t)sig.avail;
                cp_async8(&raw[buf][c][i], in ? sig.base + j : sig.base, in ? 8 : 0);
            }
        }
        cp_async_commit();
    };
    auto windowed = [&](int i0, int buf) {
#pragma unroll
        for (int m = 0; m < kFills; ++m) {
            const int e = threadIdx.x + m * kThreads;
            if (e < kCtaFrames * kTileS) {
                const int c = e / kTileS, i = e - c * kTileS;
                wx[buf][i][c] = i0 + i < window ? raw[buf][c][i] * __ldg(hann + i0 + i) : 0.0;
            }
        }
    };
    fetch(0, 0);
    cp_async_wait_all();
    __syncthreads();
    windowed(0, 0);
    if (kTileS < window) fetch(kTileS, 1);

    Cascade64 CA, CB;
    // One CTA barrier a tile. At tile t: tile t+1's copies (issued a tile
    // earlier) are waited for; behind the barrier every thread is done
    // filtering tile t-1 (whose windowed buffer tile t+1 takes) and done
    // windowing tile t (whose copy buffer tile t+2 takes); then tile t+1 is
    // windowed, tile t+2's copies are issued, and tile t is filtered.
    int buf = 0;
    for (int i0 = 0; i0 < window; i0 += kTileS) {
        const int next = i0 + kTileS;
        if (next < window) cp_async_wait_all();
        __syncthreads();
        if (next < window) windowed(next, buf ^ 1);
        if (next + kTileS < window) fetch(next + kTileS, buf);
        const int count = window - i0 < kTileS ? window - i0 : kTileS;
        filter_tile(wx[buf], q, count, k, CA, CB);
        buf ^= 1;
    }
    if (band_raw < nb && f < job.nf) {
        const double inv_n = 1.0 / (double)window;
        double *out = job.out + (int64_t)band * job.nf;
        out[f] = sqrt(CA.acc * inv_n) * k.post64;
        if (f + 1 < job.nf) out[f + 1] = sqrt(CB.acc * inv_n) * k.post64;
    }
}

}  // namespace

int gammatone_staged_frames_per_cta() { return kCtaFrames; }

void fill_fast_band_coeffs(const BandCoeffs *run, int nb, FastBandCoeffs *out) {
    for (int b = 0; b < nb; ++b) {
        const BandCoeffs &c = run[b];
        FastBandCoeffs &k = out[b];
        const double a0 = c.ca0;
        k.d1 = c.d1;
        k.d2 = c.d2;
        k.beta64[0] = c.s1n1 / c.s1n0;
        k.beta64[1] = c.s2n1 / a0;
        k.beta64[2] = c.s3n1 / a0;
        k.beta64[3] = c.s4n1 / a0;
        k.post64 = fabs(c.s1n0 * a0 * a0 * a0);
    }
}

void launch_gammatone_staged(const SpecJob *d_jobs, const void *d_tiles, int ntiles, const FastBandCoeffs *d_coeffs,
                             int nb, const double *d_hann, int window, int hop, cudaStream_t s) {
    if (ntiles <= 0) return;
    const Tile *t = static_cast<const Tile *>(d_tiles);
    if (nb > 24)
        gammatone_staged_kernel<256><<<ntiles, 256, 0, s>>>(d_jobs, t, d_coeffs, nb, d_hann, window, hop);
    else
        gammatone_staged_kernel<192><<<ntiles, 192, 0, s>>>(d_jobs, t, d_coeffs, nb, d_hann, window, hop);
    launch_counter() += 1;
}

}  // namespace vqb
