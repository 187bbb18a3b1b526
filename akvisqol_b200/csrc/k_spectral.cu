// Gammatone RMS spectrograms of the FMA forms from each frame's power
// spectrum (the cascade of reference src/gammatone.zig:268-306, without
// running it sample by sample).
//
// A band's energy over a frame, sum_{i < W} y_i^2 with y = h * x the cascade's
// response from zero state to the windowed frame x, is the energy of the
// whole response less that of its tail behind the frame:
//
//   sum_i y_i^2 = sum_k |X_k|^2 G_k / N  -  sum_{j < 8} (sum_i x_i B_j(W - i))^2
//
// * X is the frame's transform of N >= 2 W points and G_k = |H(2 pi k / N)|^2
//   (for the lowest bands, whose response would wrap around the transform,
//   the transform of h's autocorrelation cut at the window: the same sum).
// * behind the frame the cascade's eight state values decide the tail, so
//   its energy is a quadratic form of eight functionals of x; in an orthonormal
//   basis of the tails it is the sum of their squares. A functional's
//   weights decay as e^(-alpha d) with the distance d from the frame's end, so
//   only the lowest bands' reach across the whole window.
//
// All of it in f64 (the tables are formed in wider arithmetic). Against the recurrence run in extended precision the RMS
// is off by 1.3e-14 rms and 1.2e-13 at most over music, speech, low-passed
// and quantised frames and onsets, where the recurrence in f64 FMAs is off by
// 2.8e-14 and 3.5e-13: no long recurrence, and but for the lowest bands sums of
// positive terms. (Those bands' weights change sign, the autocorrelation
// being cut at the window: where a frame is one high tone cut short and the
// band 45 dB of RMS below it, 21 bands at 16 kHz, the difference is off by
// 6e-12 at most, the recurrence by 2e-12.)
//
// Work per 48 kHz frame (W = 3840, 32 bands) in f64 multiply-adds: the
// transform ~185 k, the band sums 131 k, the tails 420 k: 0.74 M, where the
// recurrence takes 14 a sample and band, 1.72 M. The two contractions run on
// the f64 tensor instruction (mma m8n8k4: the FP64 pipe's full rate, one
// instruction for 256 multiply-adds), and 32 frames are 42 independent pieces
// of work instead of 32 recurrences of 3840 steps each. Measured per 48 kHz
// frame in a launch of 2048: 28 ns for the spectrum, 43 for the band sums and
// tails (31 at the FP64 tensor rate), 5 to finish; the recurrence took 128 in
// f64 and 105 with its last two stages in f32. A single 6.4 s pair's call went
// from 1.34 ms to 0.70, 64 pairs of 10 s from 18.0 ms to 11.2.
//
// Three launches over up to 2048 48 kHz frames (a spectrum row is 33 KB; 2048
// rows stay in the L2): spectrum_kernel, a CTA per frame; energy_kernel, a warp per
// piece and tile of 32 frames; finish_kernel, the pieces added in order.
// Every frame's values are formed in the same order whatever its batch.
#include <algorithm>

#include "device.cuh"
#include "kernels.h"

namespace vqb {

namespace {

__device__ inline double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ inline double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ inline double2 cmul(double2 x, double2 w) {
    return make_double2(__fma_rn(x.x, w.x, -(x.y * w.y)), __fma_rn(x.x, w.y, x.y * w.x));
}
// x e^(-2 pi i k / 16), k < 8 (a constant once the stage loops are unrolled)
__device__ inline double2 w16(double2 x, int k) {
    constexpr double c = 0.92387953251128675613, s = 0.38268343236508977173, h = 0.70710678118654752440;
    switch (k) {
        case 0: return x;
        case 1: return cmul(x, make_double2(c, -s));
        case 2: return make_double2(h * (x.x + x.y), h * (x.y - x.x));
        case 3: return cmul(x, make_double2(s, -c));
        case 4: return make_double2(x.y, -x.x);
        case 5: return cmul(x, make_double2(-s, -c));
        case 6: return make_double2(h * (x.y - x.x), -h * (x.x + x.y));
        default: return cmul(x, make_double2(-c, -s));
    }
}

// e^(-2 pi i bitrev4(m) / 32)
__device__ inline double2 root32(int m) {
    constexpr double c[9] = {1.0, 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708,
                             0.70710678118654752440, 0.55557023301960222474, 0.38268343236508977173,
                             0.19509032201612826785, 0.0};
    const int e = (m & 1) * 8 + (m & 2) * 2 + (m & 4) / 2 + (m & 8) / 8;
    return e <= 8 ? make_double2(c[e], -c[8 - e]) : make_double2(-c[16 - e], -c[e - 8]);
}

// Radix-2 DIF stages R0 .. 3 of 16-point blocks held in registers; register m
// ends with position m of its block (bit-reversed frequency).
template <int R0>
__device__ inline void stages(double2 (&x)[16]) {
#pragma unroll
    for (int r = R0; r < 4; ++r) {
        const int half = 8 >> r;
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            if (m & half) continue;
            const double2 a = x[m], b = x[m + half];
            x[m] = cadd(a, b);
            x[m + half] = w16(csub(a, b), (m & (half - 1)) << r);
        }
    }
}

__device__ inline int padi(int e) { return e + (e >> 4); }  // 16-byte points: strides T, T / 16 and 1 without conflicts

// 4 |X_k|^2 of one frame, k = 0 .. M: the 2 M real points as M complex ones,
// z[n] = x[2n] + i x[2n + 1], M = 16 T, 16 points a thread: three register
// passes (radix 16, 16 and M / 256) with one exchange each, the deferred
// twiddles of a pass applied to its outputs; then X_k from Z_k and Z_{M-k}.
// The window fills at most half of the points: the first stage has no sums.
// Entry m T + t of the row holds the frequency of position 16 t + m (the
// weights are stored in the same order), entry M the Nyquist bin.
//
// 64 KB of exchange buffer and 128 registers leave two CTAs an SM at M =
// 4096; bound by the FP64 pipe and the exchanges' latency between barriers.
template <int LOGM>
__global__ void __launch_bounds__((1 << LOGM) / 16, 512 / ((1 << LOGM) / 16)) spectrum_kernel(
    const SpectralFrame *__restrict__ frames, const double *__restrict__ hann, const double2 *__restrict__ tw,
    double *__restrict__ power, int row, int window) {
    constexpr int M = 1 << LOGM, T = M / 16, S = T / 16;
    extern __shared__ __align__(16) double2 sm[];
    const SpectralFrame fr = frames[blockIdx.x];
    const int t = threadIdx.x;
    double2 x[16];
    if (fr.lo == 0 && fr.hi == window && (window & 1) == 0 && (reinterpret_cast<uintptr_t>(fr.p) & 15) == 0) {
        // (the same in every thread: nearly every frame, the hop being even at the usual rates)
        double2 h[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int i = 2 * (t + T * m);
            x[m] = i < window ? __ldg(reinterpret_cast<const double2 *>(fr.p + i)) : make_double2(0.0, 0.0);
            h[m] = i < window ? __ldg(reinterpret_cast<const double2 *>(hann + i)) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int m = 0; m < 8; ++m) x[m] = make_double2(x[m].x * h[m].x, x[m].y * h[m].y);
    } else {
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int i = 2 * (t + T * m);
            x[m].x = i >= fr.lo && i < fr.hi ? __ldg(fr.p + i) * __ldg(hann + i) : 0.0;
            x[m].y = i + 1 >= fr.lo && i + 1 < fr.hi ? __ldg(fr.p + i + 1) * __ldg(hann + i + 1) : 0.0;
        }
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) x[m + 8] = w16(x[m], m);
    stages<1>(x);
    {
        // W^(e t), e = bitrev4(m): four loads, the rest as products of at most
        // four of them (a table of all 15 is 61 KB and misses the L1)
        const double2 w1 = __ldg(tw + t), w2 = __ldg(tw + T + t), w4 = __ldg(tw + 2 * T + t), w8 = __ldg(tw + 3 * T + t);
        const double2 w3 = cmul(w1, w2), w5 = cmul(w1, w4), w6 = cmul(w2, w4), w7 = cmul(w3, w4);
        x[8] = cmul(x[8], w1), x[4] = cmul(x[4], w2), x[12] = cmul(x[12], w3), x[2] = cmul(x[2], w4);
        x[10] = cmul(x[10], w5), x[6] = cmul(x[6], w6), x[14] = cmul(x[14], w7), x[1] = cmul(x[1], w8);
        x[9] = cmul(x[9], cmul(w1, w8)), x[5] = cmul(x[5], cmul(w2, w8)), x[13] = cmul(x[13], cmul(w3, w8));
        x[3] = cmul(x[3], cmul(w4, w8)), x[11] = cmul(x[11], cmul(w5, w8)), x[7] = cmul(x[7], cmul(w6, w8));
        x[15] = cmul(x[15], cmul(w7, w8));
    }
#pragma unroll
    for (int m = 0; m < 16; ++m) sm[padi(t + T * m)] = x[m];
    __syncthreads();
    {
        const int j = t % S, base = t / S * T + j;
        const double2 *tw2 = tw + 4 * T;
#pragma unroll
        for (int m = 0; m < 16; ++m) x[m] = sm[padi(base + S * m)];
        stages<0>(x);
#pragma unroll
        for (int m = 1; m < 16; ++m) x[m] = cmul(x[m], __ldg(tw2 + m * S + j));
#pragma unroll
        for (int m = 0; m < 16; ++m) sm[padi(base + S * m)] = x[m];
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 16; ++m) x[m] = sm[padi(16 * t + m)];
    stages<12 - LOGM>(x);
    // Position u of frequency k pairs with the position 3 h - 1 - u of M - k, h
    // the power of two below u: within a thread for t < 2, else between
    // threads t and 3 h' - 1 - t of [h', 2 h'). The lower thread of a pair
    // takes both of its entries: half the exchange and half the twiddles.
    const int hp = t < 2 ? 2 : 1 << (31 - __clz(t)), other = 3 * hp - 1 - t;
    const bool lower = 2 * t < 3 * hp;
    if (t < 2 || !lower) {  // (its own positions: no other thread reads them before)
#pragma unroll
        for (int m = 0; m < 16; ++m) sm[padi(16 * t + m)] = x[m];
    }
    __syncthreads();
    // frequency of position 16 t + m: bitrev4(m) M / 16 behind that of 16 t,
    // so its twiddle is a 32nd root of one for m times one for t
    const double2 wt = __ldg(tw + 4 * T + 16 * S + t);
    double *out = power + (int64_t)blockIdx.x * row;
    // 2 X_k = e + o, 2 conj X_{M-k} = e - o
    auto split = [&](double2 z, double2 y, double2 w, double2 &e, double2 &o) {
        const double2 d = make_double2(z.y + y.y, y.x - z.x);  // -i (z - conj y)
        e = make_double2(z.x + y.x, z.y - y.y);
        o = cmul(d, w);
    };
    auto square = [](double re, double im) { return __fma_rn(re, re, im * im); };
    if (t < 2) {
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const int u = 16 * t + m;
            double2 e, o;
            split(x[m], sm[padi(u < 2 ? u : 3 * (1 << (31 - __clz(u))) - 1 - u)], cmul(wt, root32(m)), e, o);
            out[m * T + t] = square(e.x + o.x, e.y + o.y);
        }
    } else if (lower) {
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            double2 e, o;
            split(x[m], sm[padi(16 * other + 15 - m)], cmul(wt, root32(m)), e, o);
            out[m * T + t] = square(e.x + o.x, e.y + o.y);
            out[(15 - m) * T + other] = square(e.x - o.x, e.y - o.y);
        }
    }
    if (t == 0) {
        const double re = 2.0 * (x[0].x - x[0].y);
        out[M] = re * re;
    } else if (t < 16) {
        out[M + t] = 0.0;
    }
}

// One 8 x 8 x 4 tile product: c += a b. Lane l holds a[l / 4][l % 4],
// b[l % 4][l / 4] and c[l / 4][2 (l % 4) .. + 1].
__device__ inline void mma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// 32-byte loads (p 32-byte aligned); from the signal 16- or 8-byte ones where
// a frame starts elsewhere.
__device__ inline void load4(double (&v)[4], const double *p) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}
__device__ inline void load4_unaligned(double (&v)[4], const double *p, bool half) {
    if (half) {
        const double2 a = __ldg(reinterpret_cast<const double2 *>(p)), b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
        v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = __ldg(p + i);
    }
}

// 16 rows of the products: c += a b, a[tile] the frames' rows, b[tile] the
// operand's. Lane l's four values are rows 4 (l % 4) .. + 3, product i takes
// the i-th of every lane.
template <int NT>
__device__ inline void products(double (&c)[4][NT][2], const double (&a)[4][4], const double (&b)[NT][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n) mma(c[m][n], a[m][i], b[n][i]);
}

template <int NT>
__device__ inline void store(const double (&c)[4][NT][2], double *__restrict__ part, int cap) {
    const int lane = threadIdx.x & 31, r = lane >> 2, kk = lane & 3;
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int v = 0; v < 2; ++v) part[(int64_t)(8 * n + 2 * kk + v) * cap + 8 * m + r] = c[m][n][v];
}

// Tail functionals: NT tiles of 8 columns over 32 frames.
template <int NT>
__device__ inline void tail_task(const SpectralTask &task, const SpectralFrame *__restrict__ frames,
                                 const double *__restrict__ hann, const double *__restrict__ tails, int cap,
                                 double *__restrict__ part) {
    const int lane = threadIdx.x & 31, r = lane >> 2, kk = lane & 3;
    const double *p[4];
    int lo = 0, hi = 0x7fffffff;
    unsigned align = 0;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const SpectralFrame fr = frames[8 * m + r];
        p[m] = fr.p + 4 * kk;
        lo = max(lo, fr.lo);
        hi = min(hi, fr.hi);
        align |= (unsigned)reinterpret_cast<uintptr_t>(fr.p);
    }
    lo = __reduce_max_sync(0xffffffffu, lo);
    hi = __reduce_min_sync(0xffffffffu, hi);
    align = __reduce_or_sync(0xffffffffu, align) & 31;
    const double *b = tails + task.table + 4 * lane;
    double c[4][NT][2] = {};
    struct Step {
        double a[4][4], b[NT][4], h[4];
    } now, next;
    auto load = [&](Step &o, int s) {
        load4(o.h, hann + s + 4 * kk);
#pragma unroll
        for (int n = 0; n < NT; ++n) load4(o.b[n], b + (int64_t)(s - task.k0) * 32 + n * 128);
        if (s >= lo && s + 16 <= hi) {  // every frame of the tile holds these samples
            if (align == 0) {
#pragma unroll
                for (int m = 0; m < 4; ++m) load4(o.a[m], p[m] + s);
            } else {
#pragma unroll
                for (int m = 0; m < 4; ++m) load4_unaligned(o.a[m], p[m] + s, (align & 15) == 0);
            }
        } else {
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const int flo = frames[8 * m + r].lo, fhi = frames[8 * m + r].hi;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int k = s + 4 * kk + i;
                    o.a[m][i] = k >= flo && k < fhi ? p[m][s + i] : 0.0;
                }
            }
        }
    };
    auto multiply = [&](Step &o) {
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int i = 0; i < 4; ++i) o.a[m][i] *= o.h[i];
        products<NT>(c, o.a, o.b);
    };
    load(now, task.k0);
    for (int s = task.k0; s < task.k1; s += 32) {
        const bool more = s + 16 < task.k1;
        if (more) load(next, s + 16);
        multiply(now);
        if (!more) break;
        if (s + 32 < task.k1) load(now, s + 32);
        multiply(next);
    }
    store<NT>(c, part + (int64_t)(task.slot * 32 + task.column) * cap, cap);
}

// Spectrum entries against every band's weights, 32 frames.
template <int NT>
__device__ inline void power_task(const SpectralTask &task, const double *__restrict__ weights,
                                  const double *__restrict__ power, int row, int cap, double *__restrict__ part) {
    const int lane = threadIdx.x & 31, r = lane >> 2, kk = lane & 3;
    const double *p = power + (int64_t)r * row + 4 * kk, *b = weights + task.table + 4 * lane;
    double c[4][NT][2] = {};
    struct Step {
        double a[4][4], b[NT][4];
    } now, next;
    auto load = [&](Step &o, int s) {
#pragma unroll
        for (int m = 0; m < 4; ++m) load4(o.a[m], p + (int64_t)8 * m * row + s);
#pragma unroll
        for (int n = 0; n < NT; ++n) load4(o.b[n], b + (int64_t)(s - task.k0) * 8 * NT + n * 128);
    };
    load(now, task.k0);
    for (int s = task.k0; s < task.k1; s += 32) {
        const bool more = s + 16 < task.k1;
        if (more) load(next, s + 16);
        products<NT>(c, now.a, now.b);
        if (!more) break;
        if (s + 32 < task.k1) load(now, s + 32);
        products<NT>(c, next.a, next.b);
    }
    store<NT>(c, part + (int64_t)task.slot * 8 * NT * cap, cap);
}

// grid (groups of four 32-frame tiles, tasks: the longest first), a warp per
// task and tile: the four warps of a CTA share the task's operand through L1 and run for the
// same time; no shared memory, no barriers. Operands come in fragment order,
// 32 bytes a lane, the next 16 rows' while the current ones are multiplied.
// The FP64 pipe bounds it (16 cycles a product of 8 x 8 x 4).
template <int TAIL_TILES, int NT>
__global__ void __launch_bounds__(128, 2) energy_kernel(const SpectralFrame *__restrict__ frames, int tiles,
                                                        const SpectralTask *__restrict__ tasks,
                                                        const double *__restrict__ hann,
                                                        const double *__restrict__ weights,
                                                        const double *__restrict__ tails,
                                                        const double *__restrict__ power, int row, int cap,
                                                        double *__restrict__ tail_part,
                                                        double *__restrict__ power_part) {
    const int tile = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (tile >= tiles) return;
    const SpectralTask task = tasks[blockIdx.y];
    const int f0 = 32 * tile;
    if (task.kind == 0)
        tail_task<TAIL_TILES>(task, frames + f0, hann, tails, cap, tail_part + f0);
    else
        power_task<NT>(task, weights, power + (int64_t)f0 * row, row, cap, power_part + f0);
}

// A band's RMS by the recurrence (the operations of k_gammatone_fast.cu) for
// those of a warp's 32 frames that `which` names, eight at a time: four lanes
// a frame, one a stage, each a block of eight samples behind the one before
// it, so that a sample is four FP64 instructions of the warp (a lane that runs
// all stages issues 13, and beside another stream's tensor products each
// waits for the pipe: 200 us in place of 70 a launch of a speech batch).
// Silence in front of the first sample leaves the state at zero and is
// passed over.
__device__ __noinline__ void recurrences(unsigned which, const SpectralFrame *__restrict__ frames, int band,
                                         const double *__restrict__ hann, int window, const FastBandCoeffs &k) {
    constexpr int B = 8;
    const int lane = threadIdx.x & 31, q = lane & 3;
    const double beta = k.beta64[q], nd1 = -k.d1, nd2 = -k.d2;
    while (which) {
        unsigned mine = which;
        for (int g = lane >> 2; g > 0 && mine; --g) mine &= mine - 1;
        const SpectralFrame fr = frames[mine ? __ffs(mine) - 1 : 0];
        const int lo = max(fr.lo, 0), hi = mine ? min(fr.hi, window) : 0;
        // 32 samples of the frame over its four lanes, read 32 ahead
        double p[B], h[B], x[B], v[B] = {}, v1 = 0.0, y1 = 0.0, y2 = 0.0, acc = 0.0;
        auto fetch = [&](int i0) {
#pragma unroll
            for (int j = 0; j < B; ++j) {
                const int i = i0 + B * q + j;
                const bool in = i >= lo && i < hi;
                p[j] = in ? __ldg(fr.p + i) : 0.0;
                h[j] = in ? __ldg(hann + i) : 0.0;
            }
        };
        bool quiet = true;
        fetch(0);
        for (int i0 = 0; i0 < window + 3 * B; i0 += 4 * B) {
#pragma unroll
            for (int j = 0; j < B; ++j) {
                x[j] = p[j] * h[j];
                quiet = quiet && x[j] == 0.0;
            }
            fetch(i0 + 4 * B);
            if (__all_sync(0xffffffffu, quiet)) continue;
            for (int b = 0; b < 4; ++b) {  // stage q: samples from i0 + B (b - q)
#pragma unroll
                for (int j = 0; j < B; ++j) {
                    const double first = __shfl_sync(0xffffffffu, x[j], b, 4), before = __shfl_up_sync(0xffffffffu, v[j], 1);
                    v[j] = q ? before : first;
                }
#pragma unroll
                for (int j = 0; j < B; ++j) {
                    const double y = __fma_rn(nd1, y1, __fma_rn(nd2, y2, __fma_rn(beta, v1, v[j])));
                    v1 = v[j];
                    y2 = y1;
                    y1 = y;
                    v[j] = y;
                    if (i0 + B * (b - q) + j < window) acc = __fma_rn(y, y, acc);
                }
            }
        }
        if (q == 3 && mine) fr.out[band * fr.stride] = sqrt(acc / (double)window) * k.post64;
        for (int g = 0; g < 8 && which; ++g) which &= which - 1;
    }
}

// A thread per frame and band. Where nearly all of the response's energy
// lies behind the frame (an onset close to its end, the lowest bands) the
// difference of the two sums has lost the digits that the recurrence keeps:
// those cells, and those that are not finite, take the recurrence. At 2^-6 of
// the energy the difference has lost two digits of 1e-16, still less than the
// recurrence loses at its worst (3.5e-13); below it a few cells per onset
// remain (a pair's time and a
// batch's were the same within the runs' noise with the line at 2^-10).
constexpr double kCancelled = 1.0 / 64;
__global__ void __launch_bounds__(128) finish_kernel(const SpectralFrame *__restrict__ frames, int nframes,
                                                     const double *__restrict__ tail_part,
                                                     const double *__restrict__ power_part, int cap, int splits,
                                                     int nbp, const int32_t *__restrict__ quad_slot,
                                                     const int32_t *__restrict__ quad_segs,
                                                     const double *__restrict__ hann, int window,
                                                     const FastBandCoeffs *__restrict__ coeffs) {
    const int f = blockIdx.x * 128 + threadIdx.x, band = blockIdx.y;
    const bool inside = f < nframes;
    double total = 0.0, tail = 0.0;
    for (int s = 0; s < splits && inside; ++s) total += power_part[(int64_t)(s * nbp + band) * cap + f];
    const int slot = quad_slot[band >> 2], segs = quad_segs[band >> 2];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        double c = 0.0;
        for (int s = 0; s < segs && inside; ++s) c += tail_part[(int64_t)((slot + s) * 32 + (band & 3) * 8 + j) * cap + f];
        tail = __fma_rn(c, c, tail);
    }
    const double e = total - tail;
    const bool kept = e > kCancelled * total && e <= 1.7976931348623157e308;
    if (inside && (kept || total == 0.0)) frames[f].out[band * frames[f].stride] = kept ? sqrt(e) : 0.0;
    const unsigned rest = __ballot_sync(0xffffffffu, inside && !kept && total != 0.0);
    if (rest) recurrences(rest, frames + (f & ~31), band, hann, window, coeffs[band]);
}

constexpr int kWide = 1024;   // frames from which a tail task takes four bands

// Frames of a launch: as many as leave their spectra in the L2 (67 MB).
int chunk_frames(const SpectralTables &t) { return 2048 << (12 - t.log_m); }

}  // namespace

int spectral_scratch_frames(const SpectralTables &t, int nframes) {
    return (std::min(nframes, chunk_frames(t)) + 31) / 32 * 32;  // whole tiles
}
size_t spectral_scratch_count(const SpectralTables &t, int scratch_frames) {
    return (size_t)scratch_frames * (size_t)(t.row + 32 * t.slots + t.nbp * t.splits);
}

int spectral_frame_count(int nframes) { return (nframes + 63) / 64 * 64; }

void spectral_init_attributes() {
    cudaFuncSetAttribute(spectrum_kernel<12>, cudaFuncAttributeMaxDynamicSharedMemorySize, (4096 + 256) * 16);
}

void launch_spectral(const SpectralTables &t, const SpectralDevice &d, const FastBandCoeffs *d_coeffs,
                     const SpectralFrame *d_frames, int nframes, double *d_scratch, int scratch_frames, cudaStream_t s) {
    const int cap = scratch_frames;
    double *power = d_scratch, *tail_part = power + (size_t)cap * t.row,
           *power_part = tail_part + (size_t)cap * 32 * t.slots;
    const int M = 1 << t.log_m;
    const size_t smem = (size_t)(M + M / 16) * sizeof(double2);
    for (int f0 = 0; f0 < nframes; f0 += cap) {
        const int n = std::min(cap, nframes - f0);
        const SpectralFrame *fr = d_frames + f0;
        if (t.log_m == 12)
            spectrum_kernel<12><<<n, M / 16, smem, s>>>(fr, d.hann, d.twiddles, power, t.row, t.window);
        else if (t.log_m == 11)
            spectrum_kernel<11><<<n, M / 16, smem, s>>>(fr, d.hann, d.twiddles, power, t.row, t.window);
        else
            spectrum_kernel<10><<<n, M / 16, smem, s>>>(fr, d.hann, d.twiddles, power, t.row, t.window);
        // Four bands a tail task halve the operand traffic; two spread a small
        // launch over twice the warps. (The same sums in the same order.)
        const bool wide = n >= kWide;
        const int tiles = (n + 31) / 32;
        const dim3 grid((unsigned)((tiles + 3) / 4), (unsigned)(wide ? t.wide : t.narrow).size());
#define VQB_ENERGY(TT, NT)                                                                                          \
    energy_kernel<TT, NT><<<grid, 128, 0, s>>>(fr, tiles, TT == 4 ? d.wide : d.narrow, d.hann, d.weights, d.tails, \
                                               power, t.row, cap, tail_part, power_part)
        if (wide && t.nbp == 32)
            VQB_ENERGY(4, 4);
        else if (wide)
            VQB_ENERGY(4, 3);
        else if (t.nbp == 32)
            VQB_ENERGY(2, 4);
        else
            VQB_ENERGY(2, 3);
#undef VQB_ENERGY
        finish_kernel<<<dim3((unsigned)((n + 127) / 128), (unsigned)t.nb), 128, 0, s>>>(
            fr, n, tail_part, power_part, cap, t.splits, t.nbp, d.quad_slot, d.quad_segs, d.hann, t.window, d_coeffs);
        launch_counter() += 3;
    }
}

}  // namespace vqb
