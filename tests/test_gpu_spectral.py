"""FMA forms' spectrograms from power spectra (k_spectral.cu) where they can go
wrong: frame counts around the kernels' 32- and 64-frame tiles, hops that
leave frames unaligned, every transform size, rates whose windows keep the
recurrence, and sound that starts in a frame's last sixteenth, where the
lowest bands are recomputed by the recurrence. Cells agree with the exact form
to ~1e-13 of their RMS: MOS within 1e-10, decisions identical."""

import numpy as np
import pytest

from test_gpu_forms import check, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sr,frames", [(48000, 63), (48000, 64), (48000, 97), (22050, 65), (11025, 64), (96000, 65)])
@pytest.mark.parametrize("form", ["balanced", "fast"])
def test_onsets(native, oracle, sr, frames, form):
    window = int(np.floor(sr * 0.08 + 0.5))
    hop = window // 4
    n = window + (frames - 1) * hop + 3
    rng = np.random.default_rng(n)
    pairs = []
    for late in (window // 16, window // 40):
        start = 9 * hop + window - late
        ref = np.zeros(n)
        ref[start:] = 0.1 * rng.standard_normal(n - start) + 0.05 * np.sin(np.arange(n - start) * 0.02)
        deg = 0.8 * ref
        deg[start:] += 0.01 * rng.standard_normal(n - start)
        pairs.append((ref, deg))
    ctx = native.Context(mode=native.MODE_AUDIO, precision=form)
    check(run(ctx, pairs, sr), pairs, sr, oracle, oracle.options(), 1e-10)

