"""The gammatone's reverse where its blocks do not divide the window (3528,
1764 and 640 samples in blocks of 128, sub-blocks of 8) and where bands leave a
warp's lanes idle, against central differences of the oracle's score."""

import pytest

from test_gpu_grad import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sr,seconds", [(44100, 1.4), (22050, 1.7), (8000, 2.0)])
def test_gradient(native, oracle, sr, seconds):
    from akvisqol_b200 import synth
    ref, deg = synth.audio_pair(synth.SEED_BASE + 7, seconds=seconds, sample_rate=sr, cutoff_hz=0.3 * sr)
    check(native, oracle, ref, deg, sr, native.MODE_AUDIO, "balanced", oracle.options(), picks=4)
