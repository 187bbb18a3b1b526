"""Signals from pageable memory, staged in pieces by several threads from 16
MB on: the same scores as from device memory, at lengths around a piece (65536
samples) and around the line, twice so that the pieces are used again."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ref_len,deg_len", [(1 << 20, 1 << 20), ((1 << 20) + 1, (1 << 20) - 1), (1 << 20, (1 << 20) - 1),
                                             (1_600_000, 65537)])
def test_same_as_device_inputs(native, ref_len, deg_len):
    import torch
    rng = np.random.default_rng(ref_len + deg_len)
    ref = 0.1 * rng.standard_normal(ref_len)
    deg = np.resize(ref, deg_len) + 0.01 * rng.standard_normal(deg_len)
    ctx = native.Context(mode=native.MODE_AUDIO, precision="balanced")
    (code, host, _), = ctx.measure_batch_traced([ref], [deg], 48000)
    (_, again, _), = ctx.measure_batch_traced([ref], [deg], 48000)
    d = [torch.tensor(a, device="cuda") for a in (ref, deg)]
    torch.cuda.synchronize()
    (dcode, device, _), = ctx.measure_batch_traced([d[0].data_ptr()], [d[1].data_ptr()], 48000, device_inputs=True,
                                                   ref_lens=[ref_len], deg_lens=[deg_len])
    assert code == dcode == 0
    assert host["moslqo"] == again["moslqo"] == device["moslqo"]
    assert np.array_equal(host["fvnsim"], device["fvnsim"])
