"""The alignment DP at the sizes where its kernel changes over: 256 threads
take 1, 2, 4 or 8 slides each (rows of up to 256, 512, 1024 and 2048 slides,
then further rounds), and rows of up to 12288 slides lie in shared memory,
longer ones beside them in global memory. Identical to the CPU's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(native, oracle, sims, lo, hi):
    got, want = native.dp(sims, lo, hi), oracle.dp_backtrack(sims, lo, hi)
    assert got[2] == want[2]
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("frames", [255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2047, 2048, 2049])
@pytest.mark.parametrize("ties", [False, True])
def test_full_rows(native, oracle, frames, ties):
    rng = np.random.default_rng(frames)
    sims = rng.uniform(-0.2, 1.0, (5, frames))
    if ties:
        sims = np.round(sims, 1)
    same(native, oracle, sims, np.zeros(5, np.int64), np.full(5, frames - 1))


@pytest.mark.parametrize("ties", [False, True])
def test_held_and_global_rows(native, oracle, ties):
    """Windows of 12288, 12289, 300, 12400, 12288 and 12290 slides in turn: a
    row held in shared memory behind one in global memory, and the reverse."""
    frames = 13000
    rng = np.random.default_rng(7)
    sims = rng.uniform(-0.2, 1.0, (6, frames))
    if ties:
        sims = np.round(sims, 1)
    lo = np.array([0, 5, 100, 200, 300, 310])
    hi = lo + np.array([12288, 12289, 300, 12400, 12288, 12290]) - 1
    assert hi.max() < frames
    same(native, oracle, sims, lo, hi)
