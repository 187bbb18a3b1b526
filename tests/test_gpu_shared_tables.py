"""The FMA forms' tables of a rate lie on a device once, whatever the number of
contexts and lanes that use them."""

import pytest

pytestmark = pytest.mark.gpu

ARENA = 256 << 20  # an engine's arena after its first batch


def test_one_copy_a_device(native, monkeypatch):
    """A context of its own kind first (tables, module loading, autotuning),
    then eight more of one lane each: beyond their arenas they take less than
    2 MB each, where a copy of the tables is over 4."""
    import gc

    import torch
    from akvisqol_b200 import synth
    monkeypatch.setenv("VISQOL_GPU_LANES", "1")
    ref, deg = synth.audio_pair(synth.SEED_BASE + 980, seconds=2.0)

    def context():
        ctx = native.Context(mode=native.MODE_AUDIO, precision="balanced")
        assert ctx.measure_batch_traced([ref], [deg], 48000)[0][0] == 0
        return ctx

    held = [context()]
    gc.collect()  # no earlier context goes while the memory is counted
    free = torch.cuda.mem_get_info()[0]
    held += [context() for _ in range(8)]
    taken = free - torch.cuda.mem_get_info()[0]
    assert 8 * ARENA <= taken <= 8 * (ARENA + (2 << 20)), taken
