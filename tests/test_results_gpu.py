"""Per-cell sums and covariances at the sizes where their kernels and copies
can go wrong: cell counts around the eight a combine step loads ahead, and
results on either side of the 4 MiB from which a copy to the host is staged,
with whole and ragged last chunks."""
import numpy as np
import pytest

import tos_b200 as T
from helpers import small_catalog

pytestmark = pytest.mark.gpu

FIELDS = ("didj", "di", "dj", "wgt", "wi", "wj", "z", "num_pairs")


@pytest.mark.parametrize("nb", [50, 724, 725, 1024, 1500])
def test_subsample_covariance_sizes(engine, nb):
    rng = np.random.default_rng(nb)
    rows = np.zeros((9, nb), dtype=T.XIBIN_DTYPE)
    rows["didj"] = rng.normal(0, 1, rows.shape)
    rows["wgt"] = rng.uniform(0.5, 2, rows.shape)
    rows["num_pairs"] = 1
    xi, mean, cov = T.subsample_covariance(engine, rows)
    want = rows["didj"] / rows["wgt"]
    d = want - want.mean(axis=0)
    ref = (len(d) - 1) / len(d) * (d.T @ d)
    # nine products of FP64 values below 40: 1e-12 covers their rounding
    np.testing.assert_allclose(xi, want, rtol=1e-15)
    np.testing.assert_allclose(mean, want.mean(axis=0), rtol=0, atol=1e-13)
    np.testing.assert_allclose(cov, ref, rtol=0, atol=1e-12)


@pytest.mark.parametrize("order", [3, 5, 6, 7])
@pytest.mark.parametrize("axis", ["[0:200]*20", "[0:200]*70"])
def test_cells_add_up(engine, order, axis):
    """The total is the cells' sums added in ascending cell order, bit for bit."""
    los, px, meta = small_catalog(n=150, seed=23, size_deg=8.0, max_pixels=60)
    cat = T.Catalog(engine, los, px, order)
    bins, cells, st = T.xi_run(engine, cat, T.Grid.cartesian(axis, axis), meta["scale"], subsamples=True)
    again, _, _ = T.xi_run(engine, cat, T.Grid.cartesian(axis, axis), meta["scale"])
    cat.close()
    assert len(cells) == st["num_cells"] and bins["num_pairs"].sum() > 0
    for f in FIELDS:
        total = np.zeros_like(bins[f])
        for row in cells[f]:
            total = total + row
        assert np.array_equal(bins[f], total) and np.array_equal(bins[f], again[f])
