"""The alignment DP where its rows' split can go wrong: windows around one
slide a thread (512), several slides, more than one round of the CTA (4096),
rows too long for shared memory (12288), windows that move past the row
before, ties and equal rows. Identical to the CPU's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames,rows,radius", [(1, 1, 5), (512, 3, 9000), (513, 4, 9000), (1030, 5, 300), (4096, 3, 9000),
                                                (4097, 4, 9000), (9001, 3, 20000), (12288, 2, 20000), (12300, 3, 20000),
                                                (700, 40, 3)])
@pytest.mark.parametrize("ties", [False, True])
def test_windows(native, oracle, frames, rows, radius, ties):
    rng = np.random.default_rng(frames + rows)
    sims = rng.uniform(-0.2, 1.0, (rows, frames))
    if ties:
        sims = np.round(sims, 1)
        sims[:, frames // 2:] = 0.0
    idx = np.sort(rng.integers(0, frames, rows))
    lo = np.maximum(0, idx - radius)
    hi = np.maximum(lo, np.minimum(idx + radius, frames - 1))
    off, valid, reached = native.dp(sims, lo, hi)
    woff, wvalid, wreached = oracle.dp_backtrack(sims, lo, hi)
    assert reached == wreached
    assert np.array_equal(off, woff) and np.array_equal(valid, wvalid)


def test_sizes_in_threads(native, oracle):
    """Rows of different lengths launched by two threads at once: neither's
    shared memory is taken back by the other."""
    import functools
    import threading
    rng = np.random.default_rng(2)
    jobs = []
    for run, frames in ((native.dp, 2300), (functools.partial(native.dp, static_scratch=True), 12000)):
        sims = rng.uniform(0, 1, (4, frames))
        lo, hi = np.zeros(4, np.int64), np.full(4, frames - 1)
        jobs.append((run, sims, lo, hi, oracle.dp_backtrack(sims, lo, hi)[0]))
    wrong = []

    def work(run, sims, lo, hi, want):
        for _ in range(150):
            try:
                if not np.array_equal(run(sims, lo, hi)[0], want):
                    wrong.append("offsets")
            except Exception as e:  # noqa: BLE001
                wrong.append(repr(e))

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:3]
