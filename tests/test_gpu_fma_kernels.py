"""The FMA forms' gammatone kernels against each other and the CPU: the
recurrence on staged tiles, which serves windows above 4096 samples or up to
512, with both of its band layouts and a last tile that is not full; the power
spectra's tasks by two and by four bands (a launch of up to 1023 frames, or of
more); FAST and BALANCED, which share them."""

import numpy as np
import pytest

from test_gpu_forms import DISCRETE, check, run

pytestmark = pytest.mark.gpu

FEATURES = ("fvnsim", "fvnsim10", "fstdnsim", "fvdegenergy")


def pair(rate, seconds, seed):
    from akvisqol_b200 import synth
    return synth.audio_pair(synth.SEED_BASE + seed, seconds=seconds, sample_rate=rate, cutoff_hz=min(0.4 * rate, 7000.0))


@pytest.mark.parametrize("mode,rate,seconds", [(0, 96000, 2.3), (0, 6000, 2.3), (1, 96000, 2.3), (1, 64000, 1.7)])
def test_recurrence(native, oracle, mode, rate, seconds):
    """32 and 21 bands, 16 frames a tile. Cells are within 3.5e-13 of their
    value: 1.5e-12 dB, so the mean energies of a band agree to 1e-10 dB."""
    pairs = [pair(rate, seconds, 950 + i) for i in range(2)]
    opts = oracle.options(mode=mode)
    got = run(native.Context(mode=mode, use_lattice_model=False, precision="balanced"), pairs, rate)
    check(got, pairs, rate, oracle, opts, 1e-10)
    for (_, res, tr), (ref, deg) in zip(got, pairs):
        assert tr["nf_ref"] % 16 or tr["nf_deg"] % 16
        want, _ = oracle.measure(ref, deg, rate, opts)
        assert np.max(np.abs(res["fvdegenergy"] - want["fvdegenergy"])) <= 1e-10


@pytest.mark.parametrize("mode,rate", [(0, 48000), (0, 22050), (1, 16000)])
def test_narrow_and_wide_tasks(native, monkeypatch, mode, rate):
    """A pair of 100 frames alone and beside one of 1200: the same bits."""
    monkeypatch.setenv("VISQOL_GPU_LANES", "1")
    ctx = native.Context(mode=mode, use_lattice_model=False, precision="balanced")
    short, long = pair(rate, 2.1, 960), pair(rate, 24.0, 961)
    (code, alone, trace), = run(ctx, [short], rate)
    (code2, both, trace2), (code3, _, long_trace) = run(ctx, [short, long], rate)
    assert code == code2 == code3 == 0
    assert max(trace["nf_ref"], trace["nf_deg"]) < 1024 <= min(long_trace["nf_ref"], long_trace["nf_deg"])
    assert alone["moslqo"] == both["moslqo"]
    for key in FEATURES:
        assert np.array_equal(alone[key], both[key]), key
    for key in DISCRETE:
        assert np.array_equal(trace[key], trace2[key]), key


@pytest.mark.parametrize("mode,rate", [(0, 48000), (1, 16000), (0, 96000)])
def test_fast_equals_balanced(native, mode, rate):
    pairs = [pair(rate, 2.2 + i, 970 + i) for i in range(2)]
    fast, balanced = (run(native.Context(mode=mode, use_lattice_model=False, precision=form), pairs, rate)
                      for form in ("fast", "balanced"))
    for (c0, a, _), (c1, b, _) in zip(fast, balanced):
        assert c0 == c1 == 0
        assert a["moslqo"] == b["moslqo"]
        for key in FEATURES:
            assert np.array_equal(a[key], b[key]), key
