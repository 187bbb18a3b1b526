// Tables of the FMA forms' gammatone energies; see k_spectral.cu for
// the identity they serve. Everything is formed in long double (x87, 64-bit
// significands) or wider and rounded once.
#include "spectral_tables.h"

#include <algorithm>
#include <array>
#include <atomic>
#include <cmath>
#include <deque>
#include <mutex>
#include <thread>

#include "shared_tables.h"
#include "threads.h"

namespace vqb {

namespace {

using real = long double;
constexpr real kPi = 3.141592653589793238462643383279502884L;
constexpr int kSegment = 480;   // samples of a kind 0 task, at most
constexpr int kSplit = 512;     // spectrum entries of a kind 1 task
constexpr real kReach = 40.0L;  // a tail functional reaches back kReach / alpha samples (its weights then below e^-40 40^3 / 6 = 4.5e-14)
constexpr size_t kAnchor = 32;  // samples, a power of two
constexpr real kWrap = 50.0L;   // a band's response has died out after kWrap / alpha samples

// Quadruple precision for what the rest is derived from: the lowest bands'
// rejection of slow drifts and the difference of the two energies lose
// digits that long double does not have to spare. Only +, -, *, / and roots.
using quad = __float128;
quad root(quad v) {
    quad r = std::sqrt((real)v);
    for (int i = 0; i < 2; ++i) r = (r + v / r) / 2;
    return r;
}

using Map = std::array<std::array<quad, 8>, 8>;
Map product(const Map &a, const Map &b) {
    Map c{};
    for (int i = 0; i < 8; ++i)
        for (int k = 0; k < 8; ++k)
            if (a[i][k] != 0)
                for (int j = 0; j < 8; ++j) c[i][j] += a[i][k] * b[k][j];
    return c;
}

// The tails' orthonormal basis phi_0 .. phi_7: the Kautz functions of the pole
// pair, four times over. Section s of the chain is fed u_s, u_0 a unit impulse
// and u_{s+1} the all-pass (d2 + d1 z^-1 + z^-2) / (1 + d1 z^-1 + d2 z^-2) of
// u_s; with b = -d1 / (1 + d2), g^2 = 1 - d2^2, c^2 = 1 - b^2 it runs
//   phi_2s     <- b d2 phi_2s - c d2 phi_2s+1 + g u_s
//   phi_2s+1   <- c phi_2s + b phi_2s+1
//   u_{s+1}     = d2 u_s - b g phi_2s + c g phi_2s+1   (of the step before)
// (orthogonal maps of state and input, which is what makes the basis
// orthonormal).
struct Tails {
    Map step{};                // phi(n + 1) = step phi(n); a tail's coefficients follow the transpose
    std::array<quad, 8> at0{};  // those of h itself
    Tails(const BandCoeffs &co, const quad (&beta)[4], size_t n) {
        const quad d1 = co.d1, d2 = co.d2, b = -d1 / (1 + d2), g = root(1 - d2 * d2), c = root(1 - b * b);
        quad phi[8] = {}, gain = 1;
        for (int s = 0; s < 4; ++s, gain *= d2) {
            step[2 * s][2 * s] = b * d2, step[2 * s][2 * s + 1] = -c * d2;
            step[2 * s + 1][2 * s] = c, step[2 * s + 1][2 * s + 1] = b;
            quad through = g;
            for (int t = s - 1; t >= 0; --t, through *= d2) {
                step[2 * s][2 * t] = -through * b * g;
                step[2 * s][2 * t + 1] = through * c * g;
            }
            phi[2 * s] = g * gain;
        }
        // the cascade: p_s = u_s / D, u_{s+1}(n) = p_s(n) + beta_s p_s(n - 1);
        // state p_s(n), p_s(n - 1), all p_s(0) = 1
        Map cascade{};
        std::array<quad, 8> u{};  // u_s(n + 1) from the state at n
        for (int s = 0; s < 4; ++s) {
            cascade[2 * s] = u;
            cascade[2 * s][2 * s] -= d1, cascade[2 * s][2 * s + 1] -= d2;
            cascade[2 * s + 1][2 * s] = 1;
            u = cascade[2 * s];
            u[2 * s] += beta[s];
        }
        // h(n) = p_3(n) + beta_3 p_3(n - 1): sum of phi(n) h(n) by doubling
        Map sum{}, a = step, h = cascade;
        for (int i = 0; i < 8; ++i) sum[i][6] = phi[i], sum[i][7] = phi[i] * beta[3];
        for (size_t m = 1; m < n; m *= 2) {
            const Map more = product(product(a, sum), h);
            for (int i = 0; i < 8; ++i)
                for (int j = 0; j < 8; ++j) sum[i][j] += more[i][j];
            a = product(a, a), h = product(h, h);
        }
        for (int i = 0; i < 8; ++i) at0[i] = sum[i][0] + sum[i][2] + sum[i][4] + sum[i][6];
    }
};

struct Band {
    std::vector<real> weight;              // G_k, k = 0 .. M
    std::vector<real> tail;                // [d - 1][8]: the 8 functionals' weights of the sample d before the window's end
    size_t reach = 0;
};

// cosines: cos(2 pi k / N), k = 0 .. N - 1.
Band band_tables(const BandCoeffs &c, size_t window, size_t N, const std::vector<real> &cosines) {
    Band out;
    const real d1 = c.d1, d2 = c.d2, alpha = -0.5L * std::log(d2);
    const quad lead[4] = {(quad)c.s1n1 / c.s1n0, (quad)c.s2n1 / c.ca0, (quad)c.s3n1 / c.ca0, (quad)c.s4n1 / c.ca0};
    const real beta[4] = {(real)lead[0], (real)lead[1], (real)lead[2], (real)lead[3]};
    const real post = std::fabs((real)c.s1n0 * c.ca0 * c.ca0 * c.ca0);
    const size_t M = N / 2;
    out.reach = std::min(window, (size_t)std::ceil(kReach / alpha));
    // coefficients of the tails h(d + .), and the autocorrelation of h: of h
    // with h(d + .). From one multiple of kAnchor to the next in quad, in
    // long double between.
    const Tails tails(c, lead, (size_t)(60.0L / alpha) + 64);
    Map leap = tails.step;
    for (size_t m = 1; m < kAnchor; m *= 2) leap = product(leap, leap);
    std::array<quad, 8> anchor = tails.at0;
    real step[8][8], coef[8], a0[8];
    for (int j = 0; j < 8; ++j) {
        a0[j] = (real)anchor[j];
        for (int k = 0; k < 8; ++k) step[j][k] = (real)tails.step[j][k];
    }
    out.tail.resize(8 * window);
    std::vector<real> r(window, 0);
    for (size_t d = 0; d <= window; ++d) {
        real next[8] = {};
        if (d % kAnchor == 0) {
            std::array<quad, 8> far{};
            for (int j = 0; j < 8; ++j) {
                coef[j] = (real)anchor[j];
                for (int k = 0; k < 8; ++k) far[k] += leap[j][k] * anchor[j];
            }
            anchor = far;
        }
        for (int j = 0; j < 8; ++j) {
            if (d > 0) out.tail[8 * (d - 1) + j] = coef[j] * post / std::sqrt((real)window);
            if (d < window) r[d] += coef[j] * a0[j];
            for (int k = 0; k <= (j | 1); ++k) next[k] += step[j][k] * coef[j];
        }
        std::copy(next, next + 8, coef);
    }
    // G_k: |H|^2 where the response dies out before it wraps around the
    // transform, else the transform of the autocorrelation cut at the window
    out.weight.resize(M + 1);
    if (alpha * (real)(N - window) > kWrap) {
        // (as sums of squares: no cancellation near the poles or the zeros)
        const real rad = std::sqrt(d2), gap = (1 - d2) / (1 + rad), omega = std::atan2((real)root(d2 - (quad)d1 * d1 / 4), -d1 / 2);
        for (size_t k = 0; k <= M; ++k) {
            const real half = kPi * (real)k / (real)N, sw = std::sin(half);  // half the angle
            const real s1 = std::sin(half - omega / 2), s2 = std::sin(half + omega / 2);
            real p = 1;
            for (real bt : beta) p *= (1 + bt) * (1 + bt) - 4 * bt * sw * sw;
            const real q = (gap * gap + 4 * rad * s1 * s1) * (gap * gap + 4 * rad * s2 * s2);
            out.weight[k] = p / (q * q * q * q);
        }
    } else {
        // radix-2 transform of the even sequence, real and imaginary parts
        std::vector<real> re(N, 0), im(N, 0);
        re[0] = r[0];
        for (size_t d = 1; d < window; ++d) re[d] = re[N - d] = r[d];
        for (size_t i = 1, j = 0; i < N; ++i) {
            size_t bit = N >> 1;
            for (; j & bit; bit >>= 1) j ^= bit;
            j ^= bit;
            if (i < j) std::swap(re[i], re[j]), std::swap(im[i], im[j]);
        }
        for (size_t s = 2; s <= N; s <<= 1)
            for (size_t i = 0; i < N; i += s)
                for (size_t k = 0; k < s / 2; ++k) {
                    const size_t t = k * (N / s);
                    const real wr = cosines[t], wi = -cosines[(t + 3 * N / 4) % N];  // sin(x) = cos(x - pi/2)
                    const size_t p = i + k, q = p + s / 2;
                    const real xr = re[q] * wr - im[q] * wi, xi = re[q] * wi + im[q] * wr;
                    re[q] = re[p] - xr, im[q] = im[p] - xi;
                    re[p] += xr, im[p] += xi;
                }
        for (size_t k = 0; k <= M; ++k) out.weight[k] = re[k];
    }
    // the kernel's spectrum is 4 |X_k|^2; entries 0 < k < M stand for two
    for (size_t k = 0; k <= M; ++k)
        out.weight[k] *= post * post / (real)window * (k == 0 || k == M ? 0.25L : 0.5L) / (real)N;
    return out;
}

int bitrev(int v, int bits) {
    int r = 0;
    for (int i = 0; i < bits; ++i) r |= ((v >> i) & 1) << (bits - 1 - i);
    return r;
}

std::shared_ptr<SpectralTables> build(const std::vector<BandCoeffs> &run, size_t window) {
    auto t = std::make_shared<SpectralTables>();
    int log_m = 10;
    while (((size_t)1 << log_m) < window) ++log_m;
    const size_t M = (size_t)1 << log_m, N = 2 * M, T = M / 16;
    t->log_m = log_m;
    t->nb = (int)run.size();
    t->nbp = (t->nb + 7) / 8 * 8;
    t->window = (int)window;
    t->padded = (int)((window + 15) / 16 * 16);
    t->row = (int)M + 16;
    std::vector<real> cosines(N), sines(N);
    for (size_t k = 0; k < N; ++k) {
        cosines[k] = std::cos(2 * kPi * (real)k / (real)N);
        sines[k] = std::sin(2 * kPi * (real)k / (real)N);
    }
    cosines[N / 4] = cosines[3 * N / 4] = 0;
    std::vector<Band> bands(run.size());
    std::atomic<size_t> next{0};
    run_threads(std::min<size_t>(8, std::max(1u, std::thread::hardware_concurrency())), [&](size_t) {
        for (size_t b = next++; b < run.size(); b = next++) bands[b] = band_tables(run[b], window, N, cosines);
    });
    t->hann.assign((size_t)t->padded, 0.0);
    {
        const double denom = std::max(1.0, (double)window - 1.0);
        for (size_t i = 0; i < window; ++i) t->hann[i] = 0.5 - 0.5 * std::cos(2.0 * 3.14159265358979323846 * (double)i / denom);
    }
    // twiddles: register m of a pass carries W^(bitrev4(m) j). Pass 1: W_M^(e t)
    // for e = 1, 2, 4, 8 (the kernel multiplies the others), pass 2: all of
    // W_T^(e j), untangling: W_N^(frequency of position 16 t)
    auto unit = [&](size_t e) { return make_double2((double)cosines[e % N], (double)-sines[e % N]); };  // e^(-2 pi i e / N)
    for (size_t e = 1; e <= 8; e *= 2)
        for (size_t j = 0; j < T; ++j) t->twiddles.push_back(unit(2 * e * j));
    for (int m = 0; m < 16; ++m)
        for (size_t j = 0; j < T / 16; ++j) t->twiddles.push_back(unit(2 * 16 * (size_t)bitrev(m, 4) * j));
    for (size_t j = 0; j < T; ++j) t->twiddles.push_back(unit((size_t)bitrev((int)(16 * j), log_m)));
    // spectrum entry m T + t holds frequency bitrev(16 t + m)
    auto freq = [&](size_t s) { return (size_t)bitrev((int)(16 * (s % T) + s / T), log_m); };
    // row k and column n of an operand of `tiles` tiles
    auto at = [](size_t k, size_t n, int tiles) {
        return ((k / 16 * tiles + n / 8) * 32 + (n % 8) * 4 + k % 16 / 4) * 4 + k % 4;
    };
    // kind 1: row s for entry s of the spectrum, a column per band
    const int tiles = t->nbp / 8;
    t->weights.assign((size_t)t->row * 8 * tiles, 0.0);
    for (size_t s = 0; s <= M; ++s) {
        const size_t k = s < M ? freq(s) : M;
        for (size_t n = 0; n < run.size(); ++n) t->weights[at(s, n, tiles)] = (double)bands[n].weight[k];
    }
    std::vector<SpectralTask> spectra;
    t->splits = (int)M / kSplit;
    for (int s = 0; s < t->splits; ++s) {
        const int k0 = s * kSplit, k1 = s + 1 < t->splits ? k0 + kSplit : t->row;
        spectra.push_back(SpectralTask{1, k0, k1, k0 * 8 * tiles, s, 0});
    }
    t->wide = t->narrow = spectra;
    // kind 0: four bands from the longest one's reach to the window's end
    for (int q = 0; q < t->nb; q += 4) {
        size_t reach = 0;
        for (int n = q; n < std::min(q + 4, t->nb); ++n) reach = std::max(reach, bands[n].reach);
        const int start = (int)((window - reach) / 16 * 16);
        const int segs = (t->padded - start + kSegment - 1) / kSegment;
        const int len = ((t->padded - start) / 16 + segs - 1) / segs * 16;
        const size_t table = t->tails.size();
        t->tails.resize(table + (size_t)(t->padded - start) * 32, 0.0);
        for (int i = start; i < (int)window; ++i)
            for (int n = q; n < std::min(q + 4, t->nb); ++n)
                for (int j = 0; j < 8; ++j)
                    t->tails[table + at((size_t)(i - start), (size_t)(8 * (n - q) + j), 4)] =
                        (double)bands[n].tail[8 * (window - i - 1) + j];
        t->quad_slot.push_back(t->slots);
        t->quad_segs.push_back(segs);
        for (int s = 0; s < segs; ++s) {
            const int k0 = start + s * len, k1 = std::min(t->padded, k0 + len);
            SpectralTask task{0, k0, k1, (int)table + (k0 - start) * 32, t->slots + s, 0};
            t->wide.push_back(task);
            t->narrow.push_back(task);
            if (q + 2 < t->nb) {
                task.table += 2 * 128;
                task.column = 16;
                t->narrow.push_back(task);
            }
        }
        t->slots += segs;
    }
    auto sort = [&](std::vector<SpectralTask> &v, int tail_tiles) {
        auto cost = [&](const SpectralTask &s) { return (s.k1 - s.k0) * (s.kind ? tiles : tail_tiles); };
        std::stable_sort(v.begin(), v.end(), [&](const SpectralTask &a, const SpectralTask &b) { return cost(a) > cost(b); });
    };
    sort(t->wide, 4);
    sort(t->narrow, 2);
    return t;
}

}  // namespace

bool spectral_window(size_t window) { return window > 512 && window <= 4096; }

std::shared_ptr<const SpectralTables> spectral_tables(const std::vector<BandCoeffs> &run, size_t window) {
    // shared by the process's engines, and kept behind the last of them for
    // the next context (a program uses a few rates; the longest kept goes first)
    static SharedTables<std::vector<double>, SpectralTables> shared;
    static std::mutex mu;
    static std::deque<std::shared_ptr<const SpectralTables>> kept;
    std::vector<double> key{(double)window};
    for (const BandCoeffs &c : run)
        for (double v : {c.s1n0, c.s1n1, c.s2n1, c.s3n1, c.s4n1, c.ca0, c.d1, c.d2}) key.push_back(v);
    return shared.get(key, [&] {
        auto made = build(run, window);
        made->key = key;
        std::lock_guard<std::mutex> lock(mu);
        kept.push_back(made);
        if (kept.size() > 16) kept.pop_front();
        return made;
    });
}

}  // namespace vqb
