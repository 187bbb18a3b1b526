// Test-only: the FMA forms' frame energies from the product's tables
// (akvisqol_b200/csrc/spectral_tables.cpp) with a plain transform in long
// double, and by the recurrence in quadruple precision (its rounding grows by
// many digits where a slow drift dwarfs a low band).
#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

#include "../../akvisqol_b200/csrc/host_model.h"
#include "../../akvisqol_b200/csrc/spectral_tables.h"

using namespace vqb;

extern "C" int ss_frame(size_t nb, uint32_t rate, double high, const double *frame, size_t window, double *spectral,
                        double *recurrence) {
    using real = long double;
    if (!spectral_window(window)) return 0;
    const host::Filterbank fb = host::make_filterbank(nb, rate, 50.0, high);
    const auto t = spectral_tables(fb.run, window);
    const size_t M = (size_t)1 << t->log_m, N = 2 * M, T = M / 16;
    std::vector<real> x(window);
    for (size_t i = 0; i < window; ++i) x[i] = (real)frame[i] * t->hann[i];
    std::vector<std::complex<real>> X(x.begin(), x.end());
    X.resize(N);
    for (size_t i = 1, j = 0; i < N; ++i) {
        size_t bit = N >> 1;
        for (; j & bit; bit >>= 1) j ^= bit;
        j ^= bit;
        if (i < j) std::swap(X[i], X[j]);
    }
    const real pi = std::acos((real)-1);
    std::vector<std::complex<real>> w(N / 2);
    for (size_t k = 0; k < N / 2; ++k) w[k] = std::polar((real)1, -2 * pi * (real)k / (real)N);
    for (size_t s = 2; s <= N; s <<= 1)
        for (size_t i = 0; i < N; i += s)
            for (size_t k = 0; k < s / 2; ++k) {
                const auto a = X[i + k], b = X[i + k + s / 2] * w[k * (N / s)];
                X[i + k] = a + b;
                X[i + k + s / 2] = a - b;
            }
    const int tiles = t->nbp / 8;
    auto at = [](size_t k, size_t n, int c) {
        return ((k / 16 * c + n / 8) * 32 + n % 8 * 4 + k % 16 / 4) * 4 + k % 4;
    };
    for (size_t b = 0; b < nb; ++b) {
        real e = 0, functional[8] = {};
        for (size_t s = 0; s <= M; ++s) {
            size_t k = M;
            if (s < M) {
                k = 0;
                for (int i = 0; i < t->log_m; ++i) k |= ((16 * (s % T) + s / T) >> i & 1) << (t->log_m - 1 - i);
            }
            e += 4 * std::norm(X[k]) * t->weights[at(s, b, tiles)];
        }
        for (const SpectralTask &task : t->wide) {
            if (task.kind != 0 || task.slot < t->quad_slot[b / 4] || task.slot >= t->quad_slot[b / 4] + t->quad_segs[b / 4])
                continue;
            for (int i = task.k0; i < std::min(task.k1, (int)window); ++i)
                for (int j = 0; j < 8; ++j)
                    functional[j] += x[i] * (real)t->tails[task.table + at((size_t)(i - task.k0), b % 4 * 8 + j, 4)];
        }
        for (real f : functional) e -= f * f;
        spectral[b] = (double)std::sqrt(std::max<real>(e, 0));
        const BandCoeffs &c = fb.run[b];
        using quad = __float128;
        const quad n0[4] = {c.s1n0, c.ca0, c.ca0, c.ca0}, n1[4] = {c.s1n1, c.s2n1, c.s3n1, c.s4n1};
        quad c0[4] = {}, c1[4] = {}, sum = 0;
        for (quad v : x) {
            for (int q = 0; q < 4; ++q) {
                const quad y = n0[q] * v + c0[q];
                c0[q] = n1[q] * v + c1[q] - c.d1 * y;
                c1[q] = -c.d2 * y;
                v = y;
            }
            sum += v * v;
        }
        recurrence[b] = (double)std::sqrt((real)(sum / window));
    }
    return 1;
}
