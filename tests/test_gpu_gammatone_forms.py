"""The exact spectrogram's two kernels at either side of the rule between them
(2 x 4 x 148 warps of eight bands), at windows around their blocks of 8 and 64
samples: the CPU's bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,frames", [(8, 1184), (8, 1185), (31, 296), (31, 297), (32, 300)])
@pytest.mark.parametrize("window", [1, 7, 8, 63, 65, 130])
def test_both_kernels(native, oracle, nb, frames, window):
    coeffs, _ = oracle.filters(nb, 48000, 50.0, 24000.0)
    hop = max(1, window // 4)
    x = np.random.default_rng(window * 100 + nb).uniform(-1, 1, window + (frames - 1) * hop)
    got = native.spectrogram(x, coeffs, oracle.hann(window), window, hop)
    want = oracle.spectrogram(x, coeffs, window, hop)
    assert np.array_equal(got, want)
