"""The NSIM table and the patch statistics where their tiling can go wrong:
offsets around the 32-lane tile, band counts around the CTA's warps, patch
widths around the unrolled ones and those too wide to keep a row's cells.
Bit for bit against the oracle: the cells and the order of the sums are the
CPU's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,patch,span", [(1, 1, 1), (2, 2, 31), (3, 30, 32), (21, 20, 33), (32, 30, 65), (9, 31, 64),
                                           (8, 64, 5), (5, 65, 34), (32, 21, 40), (4, 200, 33)])
def test_table(native, oracle, nb, patch, span):
    rng = np.random.default_rng(nb * 1000 + patch)
    nfr, nfd = 2 * patch + 3, span + 7
    rs, ds = rng.uniform(0, 60, (nb, nfr)), rng.uniform(0, 60, (nb, nfd))
    ds[:, 3] = 0.0
    idx = np.array([0, 2, patch + 3])
    lo = np.array([0, 5, 6])
    hi = np.minimum(lo + span - 1, nfd - 1)
    got = native.nsim_table(rs, ds, patch, idx, lo, hi)
    want = oracle.nsim_table(rs, ds, patch, idx, lo, hi)
    for p in range(idx.size):
        assert np.array_equal(got[p, lo[p]:hi[p] + 1], want[p, lo[p]:hi[p] + 1])


@pytest.mark.parametrize("nr,nc", [(32, 32), (9, 33), (32, 64), (21, 65), (1, 31), (8, 97)])
def test_statistics(native, oracle, nr, nc):
    rng = np.random.default_rng(nr * 100 + nc)
    ref, deg = rng.uniform(0, 50, (nr, nc)), rng.uniform(0, 50, (nr, nc))
    got, want = native.patch_similarity(ref, deg), oracle.patch_similarity(ref, deg)
    assert got[0] == want[0]
    for a, b in zip(got[1:], want[1:]):
        assert np.array_equal(a, b)
