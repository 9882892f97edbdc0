"""GPU parity of the band sweep's layout for short sightlines at its edges: one
pixel up to the longest it takes and one more, short and long sightlines mixed,
item counts around its claims, and more bands than a warp owns.  Counts equal
the FP64 oracle's; sums agree to the suite's REL_TOL."""
import numpy as np
import pytest

import tos_b200 as T
from test_gap_sweep_gpu import catalog, check

pytestmark = pytest.mark.gpu

GRIDS = {
    "cartesian": lambda: T.Grid.cartesian("[0:120]*60", "[0:60]*29"),
    "observing": lambda: T.Grid.observing("[0:0.003]*70"),
}


@pytest.mark.parametrize("n_px", [1, 2, 31, 127, 128, 129])
@pytest.mark.parametrize("grid", list(GRIDS))
def test_lengths(engine, n_px, grid):
    los, px = catalog([np.arange(5 * s, 5 * s + n_px) for s in range(12)])
    _, st = check(engine, los, px, GRIDS[grid]())
    assert st["num_grid_items"] == st["num_sightline_pairs_used"] > 0


@pytest.mark.parametrize("grid", list(GRIDS))
def test_short_and_long(engine, grid):
    n = [128, 129, 3, 400, 64, 128, 1, 130, 16, 300]
    los, px = catalog([np.arange(7 * s, 7 * s + k) for s, k in enumerate(n)])
    _, st = check(engine, los, px, GRIDS[grid]())
    assert st["num_grid_items"] == st["num_sightline_pairs_used"] > 0


@pytest.mark.parametrize("n_los", [2, 3, 60])
def test_with_masked_sightlines(engine, n_los):
    kept = [np.arange(3 * s, 3 * s + 40) for s in range(n_los)]
    kept += [np.delete(np.arange(3 * s, 3 * s + 60), [11, 12, 30]) for s in range(n_los)]
    los, px = catalog(kept)
    _, st = check(engine, los, px, GRIDS["cartesian"]())
    assert 0 < st["num_grid_items"] < st["num_run_items"] == st["num_sightline_pairs_used"]


def test_many_items(engine):
    """Enough items for claims of several: equal to the pixel-pair kernel's counts."""
    rng = np.random.default_rng(5)
    los, px = catalog([rng.integers(0, 40) + np.arange(12) for _ in range(700)])
    los["ra"], los["dec"] = 3.0 + rng.random(700) * 0.02, 0.3 + rng.random(700) * 0.02
    g = T.Grid.cartesian("[0:40]*20", "[0:60]*29")
    cat = T.Catalog(engine, los, px, 6)
    bins, _, st = T.xi_run(engine, cat, g, 3586.0)
    exact, _, _ = T.xi_run(engine, cat, g, 3586.0, exact=True)
    cat.close()
    assert st["num_grid_items"] == st["num_sightline_pairs_used"] > 100000
    assert np.array_equal(bins["num_pairs"], exact["num_pairs"])
    np.testing.assert_allclose(bins["wgt"], exact["wgt"], rtol=1e-9)
