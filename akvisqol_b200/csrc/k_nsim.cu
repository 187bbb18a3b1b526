// NSIM patch similarity (reference src/nsim.zig) for the DP table and the
// per-match band statistics.
//
// Table: NSIM of every reference patch at every degraded offset in its
// search window (reference src/accel.zig:126-146, measureSimilarityAt
// src/nsim.zig:364-424). A lane owns an offset, a warp a pair of the patch's
// band rows at a time (table_kernel). Neighbouring lanes read neighbouring
// offsets of the degraded plane (coalesced) and the same reference terms.
// Interior patch columns reuse the plane's terms, whose 3x3 neighbourhood
// is the patch's; the two edge columns are recomputed with the patch's
// replicate padding, as the CPU does.
#include <algorithm>

#include "device.cuh"
#include "kernels.h"

namespace vqb {

namespace {

// sign(v) sqrt(|v|): the fast forms store variances as signed roots, so a
// cell's sqrt(srs * sds) becomes a product of two stored roots (and
// srs * sds < 0 exactly when the roots' product is negative).
__device__ inline double signed_root(double v) { return v < 0.0 ? -sqrt(-v) : sqrt(v); }

// Degraded plane of one pair: the prepared spectrogram zero-padded to
// `width` frames, its 3x3 mean and variance (reference
// src/nsim.zig:236-263).
__global__ void __launch_bounds__(256) plane_kernel(const PlaneJob *__restrict__ jobs, int nb) {
    const PlaneJob job = jobs[blockIdx.y];
    const int w = job.width, nf = job.nf;
    const int total = nb * w;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const int r = e / w, c = e - r * w;
        const int rm = r == 0 ? 0 : r - 1, rp = r + 1 >= nb ? nb - 1 : r + 1;
        const int cm = c == 0 ? 0 : c - 1, cp = c + 1 >= w ? w - 1 : c + 1;
        auto P = [&](int rr, int cc) -> double { return cc < nf ? job.spec[(int64_t)rr * nf + cc] : 0.0; };
        const double p00 = P(rm, cm), p01 = P(rm, c), p02 = P(rm, cp);
        const double p10 = P(r, cm), p11 = P(r, c), p12 = P(r, cp);
        const double p20 = P(rp, cm), p21 = P(rp, c), p22 = P(rp, cp);
        const double mu = taps9(p00, p01, p02, p10, p11, p12, p20, p21, p22);
        const double csq = taps9(p00 * p00, p01 * p01, p02 * p02, p10 * p10, p11 * p11, p12 * p12, p20 * p20,
                                 p21 * p21, p22 * p22);
        const double dms = mu * mu;
        job.pad[e] = p11;
        job.terms[e] = make_double2(mu, job.roots ? signed_root(csq - dms) : csq - dms);
    }
}

// Reference-patch terms (reference precomputeRef, src/nsim.zig:318-329):
// pairs {3x3 mean, conv(x²) - mean²}, then the patch values.
__global__ void __launch_bounds__(256) ref_terms_kernel(const RefTermsJob *__restrict__ jobs, int nb, int P) {
    const RefTermsJob job = jobs[blockIdx.y];
    const int total = nb * P;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const int r = e / P, c = e - r * P;
        const int rm = r == 0 ? 0 : r - 1, rp = r + 1 >= nb ? nb - 1 : r + 1;
        const int cm = c == 0 ? 0 : c - 1, cp = c + 1 >= P ? P - 1 : c + 1;
        auto R = [&](int rr, int cc) -> double { return job.spec[(int64_t)rr * job.nf + job.col + cc]; };
        const double p00 = R(rm, cm), p01 = R(rm, c), p02 = R(rm, cp);
        const double p10 = R(r, cm), p11 = R(r, c), p12 = R(r, cp);
        const double p20 = R(rp, cm), p21 = R(rp, c), p22 = R(rp, cp);
        const double mu = taps9(p00, p01, p02, p10, p11, p12, p20, p21, p22);
        const double csq = taps9(p00 * p00, p01 * p01, p02 * p02, p10 * p10, p11 * p11, p12 * p12, p20 * p20,
                                 p21 * p21, p22 * p22);
        const double rms = mu * mu;
        reinterpret_cast<double2 *>(job.out)[e] = make_double2(mu, job.roots ? signed_root(csq - rms) : csq - rms);
        job.out[2 * total + e] = p11;
    }
}

// The fast forms' 3x3 window as an FMA chain and their quotient: the cell's
// two quotients as one, (2 mr md + c1)(srd + c3) / ((rms + dms + c1)
// (sqrt(srs sds) + c3)), by a positive denominator with a reciprocal estimate
// refined by Newton-Raphson iterations (Markstein's refinement: r' = r +
// r(1 - d r), then q' = q + r'(n - d q)), which agrees with the IEEE quotient
// to about an ulp.
__device__ inline double taps9_fma(double a00, double a01, double a02, double a10, double a11, double a12,
                                   double a20, double a21, double a22) {
    double t = kW0 * a00;
    t = __fma_rn(kW1, a01, t);
    t = __fma_rn(kW0, a02, t);
    t = __fma_rn(kW1, a10, t);
    t = __fma_rn(kW2, a11, t);
    t = __fma_rn(kW1, a12, t);
    t = __fma_rn(kW0, a20, t);
    t = __fma_rn(kW1, a21, t);
    return __fma_rn(kW0, a22, t);
}

__device__ inline double fast_quotient(double n, double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    r = __fma_rn(r, __fma_rn(-d, r, 1.0), r);
    r = __fma_rn(r, __fma_rn(-d, r, 1.0), r);
    const double q = n * r;
    return __fma_rn(r, __fma_rn(-d, q, n), q);
}

// sr, sd: signed roots of the reference and degraded variances.
__device__ inline double sim_cell_quick(double mr, double sr, double md, double sd, double crd) {
    const double mrd = mr * md;
    const double srd = crd - mrd;
    const double q = sr * sd;
    const double sden = q < 0.0 ? kC3 : fabs(q) + kC3;
    return fast_quotient(__fma_rn(2.0, mrd, kC1) * (srd + kC3), __fma_rn(mr, mr, __fma_rn(md, md, kC1)) * sden);
}

template <bool kFast>
__device__ inline double taps(double a00, double a01, double a02, double a10, double a11, double a12, double a20,
                              double a21, double a22) {
    return kFast ? taps9_fma(a00, a01, a02, a10, a11, a12, a20, a21, a22)
                 : taps9(a00, a01, a02, a10, a11, a12, a20, a21, a22);
}

// One patch column of the ref x deg products, of the form's window.
template <bool kFast>
struct Column;
// Exact: rows r-1 .. r+1 with the window's weights applied (outer rows take kW0
// at the sides and kW1 in the centre, the middle row kW1 and kW2), summed
// in taps9's order.
template <>
struct Column<false> {
    double a, b, c;
    __device__ inline void set(double x, double y, double z, double) { a = x, b = y, c = z; }
    __device__ static inline double upper(const Column &l, const Column &m, const Column &r) {
        return taps9(l.a, m.a, r.a, l.b, m.b, r.b, l.c, m.c, r.c);
    }
    __device__ static inline double lower(const Column &, const Column &, const Column &) { return 0.0; }
};
// Fast: rows r-1 .. r+2, for the windows of rows r and r+1: the outer rows'
// sum and the middle row of each.
template <>
struct Column<true> {
    double eu, mu, el, ml;
    __device__ inline void set(double a, double b, double c, double d) { eu = a + c, mu = b, el = b + d, ml = c; }
    __device__ static inline double window(double el, double em, double er, double ml, double mm, double mr) {
        return __fma_rn(kW2, mm, __fma_rn(kW1, (ml + mr) + em, kW0 * (el + er)));
    }
    __device__ static inline double upper(const Column &l, const Column &m, const Column &r) {
        return window(l.eu, m.eu, r.eu, l.mu, m.mu, r.mu);
    }
    __device__ static inline double lower(const Column &l, const Column &m, const Column &r) {
        return window(l.el, m.el, r.el, l.ml, m.ml, r.ml);
    }
};

constexpr int kTableWarps = 8;
constexpr int kTableKept = 64;  // exact form: patch columns up to which a row's cells are kept (128 KB a CTA)

__device__ inline void hand_over(int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }
__device__ inline void take_over(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

// The table: grid (tiles of 32 offsets, patches), a lane an offset, the
// patch's band rows to the CTA's warps in turn.
//
// Exact form: the CPU adds the cells one by one in row-major order, so a warp
// keeps a row's cells in shared memory and adds them to the running sum
// when the row before has been added (a named barrier hands the 32 sums from
// warp to warp): the serial part is the additions alone, and the cells (two
// IEEE quotients and a root each) are formed by eight warps at once. Patches
// too wide to keep run on one warp. The fast forms take rows by pairs (four
// rows' products instead of six, two independent cells) and add up a warp's
// cells, then the warps.
//
// A cell is ~600 cycles of dependent quotients, roots and sums, so the warps
// in flight decide a small launch and issue slots (half of them not FP64) a
// large one: 128 registers for two CTAs an SM; by pairs the exact form has
// 190 and is slower. Against a thread per patch and offset over all its cells:
// an exact pair of 16 patches x 497 offsets 312 to 71 us, a fast one of 317
// offsets 123 to 23 us; lanes' time over 64 fast 10 s pairs 5.5 to 1.9 ms,
// over 32 exact ones 7.2 to 2.6 ms; 100 patches x 2977 offsets, which filled
// the chip before, 1.53 to 1.54 ms.
template <bool kFast, int kP>
__global__ void __launch_bounds__(kTableWarps * 32, 2) table_kernel(const TableTask *__restrict__ tasks,
                                                                      int nb, int P_) {
    const int P = kP ? kP : P_;
    extern __shared__ double cells_sm[];  // exact form: [warp][P][32]
    __shared__ double sums_sm[kTableWarps][32];
    const TableTask t = tasks[blockIdx.y];
    const int off0 = t.lo + blockIdx.x * 32;
    if (off0 > t.hi) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int off = min(off0 + lane, t.hi);
    constexpr int step = kFast ? 2 : 1;
    const int items = (nb + step - 1) / step;
    const int w = t.width;
    const double2 *rterms = reinterpret_cast<const double2 *>(t.ref_terms);
    const double *rvals = t.ref_terms + 2 * (int64_t)nb * P;
    double *mine = cells_sm + (int64_t)warp * P * 32 + lane;
    double sum = 0.0;
    for (int item = warp; item < items; item += warps) {
        const int r = item * step;
        const bool two = kFast && r + 1 < nb;
        const int rows[4] = {max(r - 1, 0), r, min(r + 1, nb - 1), min(r + 2, nb - 1)};
        const double *q[4], *p[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            q[k] = rvals + (int64_t)rows[k] * P;
            p[k] = t.pad + (int64_t)rows[k] * w + off;
        }
        const double2 *ru = rterms + (int64_t)r * P, *rl = rterms + (int64_t)rows[2] * P;
        const double2 *du = t.terms + (int64_t)r * w + off, *dl = t.terms + (int64_t)rows[2] * w + off;
        auto product = [&](int k, int c) { return __ldg(q[k] + c) * __ldg(p[k] + c); };
        auto column = [&](int c) {
            Column<kFast> v;
            v.set(product(0, c), product(1, c), product(2, c), kFast ? product(3, c) : 0.0);
            return v;
        };
        // the edge columns' mean and variance, with the patch's padding
        auto edge = [&](const double *pm, const double *p0, const double *pp, int c) {
            const int cm = max(c - 1, 0), cp = min(c + 1, P - 1);
            const double d00 = pm[cm], d01 = pm[c], d02 = pm[cp];
            const double d10 = p0[cm], d11 = p0[c], d12 = p0[cp];
            const double d20 = pp[cm], d21 = pp[c], d22 = pp[cp];
            const double md = taps<kFast>(d00, d01, d02, d10, d11, d12, d20, d21, d22);
            const double sq = taps<kFast>(d00 * d00, d01 * d01, d02 * d02, d10 * d10, d11 * d11, d12 * d12, d20 * d20,
                                          d21 * d21, d22 * d22);
            const double var = sq - md * md;
            return make_double2(md, kFast ? signed_root(var) : var);
        };
        auto cell = [&](double2 ref, double2 deg, double crd) {
            return kFast ? sim_cell_quick(ref.x, ref.y, deg.x, deg.y, crd)
                         : sim_cell(ref.x, ref.x * ref.x, ref.y, deg.x, deg.x * deg.x, deg.y, crd);
        };
        auto put = [&](int c, double u, double l) {
            if (kFast)
                sum += two ? u + l : u;
            else if (warps == 1)
                sum += u;
            else
                mine[c * 32] = u;
        };
        auto lower = [&](double2 deg, int c, const Column<kFast> &left, const Column<kFast> &mid, const Column<kFast> &right) {
            return kFast ? cell(__ldg(rl + c), deg, Column<kFast>::lower(left, mid, right)) : 0.0;
        };
        Column<kFast> left = column(0), mid = left;
        double2 mu = edge(p[0], p[1], p[2], 0), ml = kFast ? edge(p[1], p[2], p[3], 0) : mu;
#pragma unroll (kP && !kFast ? 5 : 3)
        for (int c = 0; c + 1 < P; ++c) {  // (unrolled: the columns' registers rotate without moves)
            const Column<kFast> right = column(c + 1);
            const double2 nu = __ldg(du + c + 1), nl = kFast ? __ldg(dl + c + 1) : nu;
            put(c, cell(__ldg(ru + c), mu, Column<kFast>::upper(left, mid, right)),
                lower(ml, c, left, mid, right));
            left = mid;
            mid = right;
            mu = nu;
            ml = nl;
        }
        if (P > 1) {
            mu = edge(p[0], p[1], p[2], P - 1);
            ml = kFast ? edge(p[1], p[2], p[3], P - 1) : mu;
        }
        put(P - 1, cell(__ldg(ru + P - 1), mu, Column<kFast>::upper(left, mid, mid)),
            lower(ml, P - 1, left, mid, mid));
        if (!kFast && warps > 1) {
            if (item > 0) {
                take_over(1 + warp);
                sum = sums_sm[0][lane];
            }
#pragma unroll 4
            for (int c = 0; c < P; ++c) sum += mine[c * 32];
            if (item + 1 < items) {
                sums_sm[0][lane] = sum;
                __threadfence_block();
                hand_over(1 + (warp + 1) % warps);
            }
        }
    }
    if (kFast) {
        sums_sm[warp][lane] = sum;
        __syncthreads();
        if (warp) return;
        for (int k = 1; k < warps; ++k) sum += sums_sm[k][lane];
    } else if (warp != (items - 1) % warps) {
        return;
    }
    if (off0 + lane <= t.hi) t.out[off] = sum / (double)(nb * P);
}

// Per-band statistics of one patch pair (reference measurePatchSimilarity,
// src/nsim.zig:427-510). A CTA a patch: its warps form the cells (and the
// degraded values) of 32 columns at a time, a warp a row, a lane a column, each
// from its 3x3 neighbourhood; then warp 0 adds them in the CPU's column order,
// a lane a row. Up to kStatsCache columns the cells are kept for the variance
// pass, beyond it they are formed again (same operations, same bits).
// A thread that formed its whole row alone took 28-40 us for a pair's
// patches, 120 us a launch of a batch; now 7 and 14.
constexpr int kStatsCache = 64;
constexpr int kStatsWarps = 8;

__global__ void __launch_bounds__(kStatsWarps * 32) stats_kernel(const StatsJob *__restrict__ jobs, int nb) {
    const StatsJob job = jobs[blockIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ double means_sm[32];
    __shared__ double cells_sm[kStatsCache][33];  // [column][row]
    __shared__ double deg_sm[32][33];
    int deg_col = job.deg_col;
    bool valid = true, reached = true;
    if (job.dp_offset) {
        const int64_t o = *job.dp_offset;
        reached = o >= 0;
        valid = *job.dp_valid != 0;
        deg_col = (int)(o < 0 ? 0 : o);
    }
    const int nc = job.ncols;
    if (!reached) {
        // Patches the backtrack never reached keep zeroed statistics.
        if (threadIdx.x < nb) job.means[threadIdx.x] = job.stddevs[threadIdx.x] = job.energy[threadIdx.x] = 0.0;
        if (threadIdx.x == 0) *job.similarity = 0.0;
        return;
    }
    auto R = [&](int rr, int cc) -> double { return __ldg(job.ref + (int64_t)rr * job.ref_stride + job.ref_col + cc); };
    auto D = [&](int rr, int cc) -> double {
        return deg_col + cc < job.deg_cols ? __ldg(job.deg + (int64_t)rr * job.deg_stride + deg_col + cc) : 0.0;
    };
    auto form = [&](int c0, int at) {  // columns c0 .. c0 + 31 into cells_sm[at ..]
        const int c = c0 + lane;
        if (c >= nc) return;
        for (int r = warp; r < nb; r += kStatsWarps) {
            const int rm = r == 0 ? 0 : r - 1, rp = r + 1 >= nb ? nb - 1 : r + 1;
            const int cm = c == 0 ? 0 : c - 1, cp = c + 1 >= nc ? nc - 1 : c + 1;
            const double r00 = R(rm, cm), r01 = R(rm, c), r02 = R(rm, cp), r10 = R(r, cm), r11 = R(r, c),
                         r12 = R(r, cp), r20 = R(rp, cm), r21 = R(rp, c), r22 = R(rp, cp);
            const double d00 = D(rm, cm), d01 = D(rm, c), d02 = D(rm, cp), d10 = D(r, cm), d11 = D(r, c),
                         d12 = D(r, cp), d20 = D(rp, cm), d21 = D(rp, c), d22 = D(rp, cp);
            const double mr = taps9(r00, r01, r02, r10, r11, r12, r20, r21, r22);
            const double md = taps9(d00, d01, d02, d10, d11, d12, d20, d21, d22);
            const double crs = taps9(r00 * r00, r01 * r01, r02 * r02, r10 * r10, r11 * r11, r12 * r12, r20 * r20,
                                     r21 * r21, r22 * r22);
            const double cds = taps9(d00 * d00, d01 * d01, d02 * d02, d10 * d10, d11 * d11, d12 * d12, d20 * d20,
                                     d21 * d21, d22 * d22);
            const double crd = taps9(r00 * d00, r01 * d01, r02 * d02, r10 * d10, r11 * d11, r12 * d12, r20 * d20,
                                     r21 * d21, r22 * d22);
            const double rms = mr * mr, dms = md * md;
            cells_sm[at + lane][r] = sim_cell(mr, rms, crs - rms, md, dms, cds - dms, crd);
            deg_sm[lane][r] = d11;
        }
    };
    const bool adds = warp == 0 && lane < nb, kept = nc <= kStatsCache;
    const double inv_ncols = 1.0 / (double)nc;
    double deg_sum = 0.0, sim_sum = 0.0;
    for (int c0 = 0; c0 < nc; c0 += 32) {
        const int at = kept ? c0 : 0, count = min(32, nc - c0);
        form(c0, at);
        __syncthreads();
        if (adds)
            for (int c = 0; c < count; ++c) {
                deg_sum += deg_sm[c][lane];
                sim_sum += cells_sm[at + c][lane];
            }
        __syncthreads();
    }
    const double mean = sim_sum * inv_ncols;
    double ss = 0.0;
    for (int c0 = 0; nc > 1 && c0 < nc; c0 += 32) {
        const int at = kept ? c0 : 0, count = min(32, nc - c0);
        if (!kept) {
            form(c0, 0);
            __syncthreads();
        }
        if (adds)
            for (int c = 0; c < count; ++c) {
                const double diff = cells_sm[at + c][lane] - mean;
                ss += diff * diff;
            }
        if (!kept) __syncthreads();
    }
    if (warp) return;
    if (adds) {
        job.energy[lane] = deg_sum * inv_ncols;
        job.stddevs[lane] = nc > 1 ? sqrt(ss / ((double)nc - 1.0)) : 0.0;
        job.means[lane] = valid ? mean : 0.0;
        means_sm[lane] = mean;
    }
    __syncwarp();
    if (lane == 0) {
        double acc = 0.0;
        for (int b = 0; b < nb; ++b) acc += means_sm[b];
        *job.similarity = valid ? acc / (double)nb : 0.0;
    }
}

// fast_quotient over arrays (its direct test against IEEE division).
__global__ void quotient_kernel(const double *__restrict__ num, const double *__restrict__ den,
                                double *__restrict__ out, size_t count) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
        out[i] = fast_quotient(num[i], den[i]);
}

}  // namespace

void launch_plane(const PlaneJob *d_jobs, int njobs, int nb, int max_width, cudaStream_t s) {
    if (njobs <= 0) return;
    const int total = nb * max_width;
    int blocks = (total + 255) / 256;
    if (blocks > 1024) blocks = 1024;
    plane_kernel<<<dim3((unsigned)blocks, (unsigned)njobs), 256, 0, s>>>(d_jobs, nb);
    launch_counter() += 1;
}

void launch_ref_terms(const RefTermsJob *d_jobs, int njobs, int nb, int P, cudaStream_t s) {
    if (njobs <= 0) return;
    const int total = nb * P;
    const int blocks = (total + 255) / 256;
    ref_terms_kernel<<<dim3((unsigned)blocks, (unsigned)njobs), 256, 0, s>>>(d_jobs, nb, P);
    launch_counter() += 1;
}

void nsim_init_attributes() {
    const int bytes = kTableWarps * kTableKept * 32 * (int)sizeof(double);
    cudaFuncSetAttribute(table_kernel<false, 30>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    cudaFuncSetAttribute(table_kernel<false, 20>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    cudaFuncSetAttribute(table_kernel<false, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

void launch_table(const TableTask *d_tasks, int ntasks, int max_offsets, int nb, int P, bool fast, cudaStream_t s) {
    const unsigned tiles = (unsigned)((max_offsets + 31) / 32);
    const bool kept = !fast && P <= kTableKept;
    const unsigned threads = fast || kept ? kTableWarps * 32 : 32;
    const size_t smem = kept ? (size_t)kTableWarps * P * 32 * sizeof(double) : 0;
    for (int t0 = 0; t0 < ntasks; t0 += 65535) {
        const dim3 grid(tiles, (unsigned)std::min(ntasks - t0, 65535));
        const TableTask *t = d_tasks + t0;
        // (the patch widths of the two modes as constants: loads at fixed
        // distances; 3.06 to 2.64 ms of a batch of 32 exact audio pairs)
        if (fast && P == 30)
            table_kernel<true, 30><<<grid, threads, smem, s>>>(t, nb, P);
        else if (fast && P == 20)
            table_kernel<true, 20><<<grid, threads, smem, s>>>(t, nb, P);
        else if (fast)
            table_kernel<true, 0><<<grid, threads, smem, s>>>(t, nb, P);
        else if (P == 30)
            table_kernel<false, 30><<<grid, threads, smem, s>>>(t, nb, P);
        else if (P == 20)
            table_kernel<false, 20><<<grid, threads, smem, s>>>(t, nb, P);
        else
            table_kernel<false, 0><<<grid, threads, smem, s>>>(t, nb, P);
        launch_counter() += 1;
    }
}

void launch_stats(const StatsJob *d_jobs, int njobs, int nb, cudaStream_t s) {
    if (njobs <= 0) return;
    stats_kernel<<<njobs, kStatsWarps * 32, 0, s>>>(d_jobs, nb);
    launch_counter() += 1;
}

void launch_fast_quotient(const double *num, const double *den, double *out, size_t count, cudaStream_t s) {
    if (count == 0) return;
    const size_t blocks = std::min<size_t>((count + 255) / 256, 4096);
    quotient_kernel<<<(unsigned)blocks, 256, 0, s>>>(num, den, out, count);
    launch_counter() += 1;
}

}  // namespace vqb
