// Host tables of the FMA forms' gammatone spectrograms (k_spectral.cu).
#pragma once

#include <cstddef>
#include <cstdint>
#include <memory>
#include <vector>

#include <cuda_runtime.h>

#include "device.cuh"

namespace vqb {

// One warp's share of the energy sums of 32 frames: operand tiles of 8 columns.
struct SpectralTask {
    int32_t kind;    // 0: the tail functionals of four bands (8 columns each) or of two of them; 1: all bands' weights
    int32_t k0, k1;  // samples (kind 0) or spectrum entries (kind 1), multiples of 16
    int32_t table;   // doubles into the kind's table at k0
    int32_t slot;    // partial-sum slot
    int32_t column;  // first column in the slot
};

// Everything that depends on the filterbank and the window alone.
struct SpectralTables {
    std::vector<double> key;  // what they depend on: the window and the bands' coefficients
    int log_m = 0;        // complex transform size M = 2^log_m, M >= window
    int nb = 0, nbp = 0;  // bands, padded to a multiple of 8
    int window = 0;
    int padded = 0;       // window padded to a multiple of 16
    int row = 0;          // spectrum entries of a frame's row (M + 1, padded to a multiple of 16)
    int splits = 0;       // kind 1 slots
    int slots = 0;        // kind 0 slots (32 columns each)
    std::vector<double> hann;       // `padded` values, zero past the window
    std::vector<double2> twiddles;  // pass 1 [4][M/16], pass 2 [16][M/256], untangling [M/16]
    // operands in fragment order, per 16 rows k: [column tiles][32 lanes][4],
    // lane l holding column l / 4 of rows 4 (l % 4) .. + 3
    std::vector<double> weights;  // kind 1, nbp / 8 tiles
    std::vector<double> tails;    // kind 0, per four bands their four tiles
    std::vector<int32_t> quad_slot, quad_segs;  // per four bands: their slots
    std::vector<SpectralTask> wide, narrow;     // tasks by four and by two bands, longest first
};

// Windows the transform kernels serve (1024, 2048 and 4096 points).
bool spectral_window(size_t window);
// run: the bands' coefficients (reference src/gammatone.zig:268-306).
std::shared_ptr<const SpectralTables> spectral_tables(const std::vector<BandCoeffs> &run, size_t window);

}  // namespace vqb
