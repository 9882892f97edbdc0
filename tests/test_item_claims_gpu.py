"""GPU parity where a sweep owns few of the sightline pairs and goes through the
others in growing claims: one masked sightline among contiguous ones, one
contiguous among masked ones, and Polar pairs of constant z index among pairs
whose index varies, at pair counts around the claims of 32.  Counts equal the
FP64 oracle's; sums agree to the suite's REL_TOL."""
import numpy as np
import pytest

import tos_b200 as T
from helpers import assert_counts_equal, assert_sums_close
from oracle import oracle
from test_gap_sweep_gpu import catalog

pytestmark = pytest.mark.gpu


def check(engine, los, px, g):
    cat = T.Catalog(engine, los, px, 6)
    bins, _, st = T.xi_run(engine, cat, g, 3586.0)
    cat.close()
    ref = oracle.xi(los, px, 6, g.type, g.axes_array(), 3586.0, mode=1)[0]
    ref_abs = oracle.xi(los, px, 6, g.type, g.axes_array(), 3586.0, mode=2)[0]
    assert_counts_equal(bins, ref)
    assert_sums_close(bins, ref, ref_abs)
    return st


GRIDS = {
    "cartesian": lambda: T.Grid.cartesian("[0:120]*30", "[0:60]*29"),
    "observing": lambda: T.Grid.observing("[0:0.01]*33"),
}


@pytest.mark.parametrize("n_los", [2, 8, 9, 12, 33, 64])
@pytest.mark.parametrize("odd", ["first", "last"])
@pytest.mark.parametrize("masked", [True, False])  # the odd one out
@pytest.mark.parametrize("grid", list(GRIDS))
def test_one_of_many(engine, n_los, odd, masked, grid):
    kept = []
    for s in range(n_los):
        k = 3 * s + np.arange(60)
        if (s == (0 if odd == "first" else n_los - 1)) == masked:
            k = np.delete(k, [20, 21, 40])
        kept.append(k)
    los, px = catalog(kept)
    st = check(engine, los, px, GRIDS[grid]())
    assert st["num_run_items"] == st["num_sightline_pairs_used"] > 0
    if masked and n_los > 2:
        assert 0 < st["num_grid_items"] < st["num_run_items"]
    else:
        assert st["num_grid_items"] == 0


@pytest.mark.parametrize("n_los", [36, 60])
def test_polar_mixed_z(engine, n_los):
    """The z index changes at grid value 100: pairs below it, above it and across."""
    los, px = catalog([np.arange(3 * s, 3 * s + 50) for s in range(n_los)])
    st = check(engine, los, px, T.Grid.polar("[0:150]*37", "[0:1]*11", "[1.602:3.8]*2"))
    assert 0 < st["num_diag_items"] < st["num_sightline_pairs_used"]
