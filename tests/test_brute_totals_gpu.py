"""The brute-force count's sums where one bin takes every pair of many short
lines: the total in fixed point passes what a carry-free pair of words holds
(8 points a line: above 2^36 pairs).  Unit weights and signals, so the sums are
the pair counts exactly."""
import numpy as np
import pytest

import tos_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_lines", [32768, 46000, 60000])
@pytest.mark.parametrize("nbins", [1, 4096])
def test_one_bin_takes_all(engine, n_lines, nbins):
    z = np.arange(8, dtype=np.float32)
    side = 250
    line = np.arange(n_lines)
    pts = np.ones((n_lines, 8, 5), dtype=np.float32)
    pts[..., 0] = (4 * (line % side))[:, None]
    pts[..., 1] = (4 * (line // side))[:, None]
    pts[..., 2] = z
    pts[..., 3] = -1.0
    ds, ws, ct, _ = T.brute_run(engine, pts.reshape(-1, 5), 0.0, 0.25, nbins)  # every pair is beyond the range
    n = n_lines * 8
    assert ct[nbins + 1] == n * (n - 1) // 2 and ct[:nbins + 1].sum() == 0
    assert ws[nbins + 1] == n * (n - 1) // 2 and ds[nbins + 1] == n * (n - 1) // 2
