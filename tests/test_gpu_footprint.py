"""A pair's footprint, the unit of the server's HBM admission, bounds what the
pair takes of a lane's arena, with what can make it take more: lag searches
that the f32 pass leaves undecided (their exact reruns), a degraded signal that
the alignment makes longer than its length told, realigned patches off the
frame grid, signals of a few frames. And the spectra's scratch, sized before
the lag is known, gives the same bits when it takes several passes."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def signals(kind, n):
    rng = np.random.default_rng(n)
    if kind == "constant":  # every lag alike
        return np.full(n, 0.25), np.full(n + 100, 0.25)
    if kind == "clicks":  # equal peaks a period apart
        deg = np.zeros(n + 4000)
        deg[::2000] = 0.5
        return deg[:n].copy(), np.roll(deg, 11)
    ref = 0.1 * rng.standard_normal(n)
    if kind == "late":  # the degraded signal starts near the middle: nearly half of the reference is put before it
        cut = int(0.45 * n)
        return ref, np.concatenate([ref[cut:], 0.01 * rng.standard_normal(cut // 3)])
    parts = []  # "slips": seven samples more every half second
    for i in range(0, n, n // 8):
        parts += [ref[i:i + n // 8], np.zeros(7)]
    return ref, np.concatenate(parts)


@pytest.fixture(scope="module")
def contexts(native):
    return {(form, mode): native.Context(mode=mode, use_lattice_model=False, precision=form)
            for form in ("exact", "balanced") for mode in (native.MODE_AUDIO, native.MODE_SPEECH)}


@pytest.mark.parametrize("form", ["exact", "balanced"])
@pytest.mark.parametrize("mode,rate,seconds", [(0, 48000, 0.3), (0, 8000, 1.1), (0, 48000, 1.1), (0, 44100, 10.0),
                                               (0, 48000, 22.0), (1, 16000, 0.16), (1, 16000, 0.3), (1, 16000, 1.1),
                                               (1, 16000, 15.0)])
def test_bounds_the_arena(native, contexts, form, mode, rate, seconds):
    ctx = contexts[(form, mode)]
    for kind in ("constant", "clicks", "late", "slips"):
        ref, deg = signals(kind, int(seconds * rate))
        ctx.measure_batch_traced([ref], [deg], rate)
        used = ctx.last_batch_bytes()
        assert 0 < used <= native.pair_footprint(ref.size, deg.size, rate, mode), (kind, used)


@pytest.mark.parametrize("mode,rate", [(0, 16000), (1, 16000)])
def test_passes_give_the_same_bits(native, monkeypatch, mode, rate):
    """The pair alone, whose scratch holds fewer frames than its aligned
    degraded signal has, and beside a longer one, whose frames make it larger."""
    monkeypatch.setenv("VISQOL_GPU_LANES", "1")
    ctx = native.Context(mode=mode, use_lattice_model=False, precision="balanced")
    ref, deg = signals("late", 4 * rate)
    long_ref, long_deg = signals("slips", 13 * rate)
    (code, alone, trace), = ctx.measure_batch_traced([ref], [deg], rate)
    (code2, both, _), _ = ctx.measure_batch_traced([ref, long_ref], [deg, long_deg], rate)
    assert code == code2 == 0
    assert trace["nf_deg"] > (trace["nf_ref"] + 16 + 31) // 32 * 32  # more than the scratch's frames
    assert alone["moslqo"] == both["moslqo"]
    for key in ("fvnsim", "fvnsim10", "fstdnsim", "fvdegenergy"):
        assert np.array_equal(alone[key], both[key]), key
