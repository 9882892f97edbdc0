"""GPU parity of the Polar sweep that bins pair by pair (short or uneven
sightlines, fine bins) at its edges: lengths around its 32 diagonals and the
longest it takes beside the block sweep, short and long sightlines mixed (the
block sweep's own edges among them), masked and unlike sightlines of any length
on grids to which blocks do not suit.  Counts equal the FP64 oracle's; sums agree
to the suite's REL_TOL."""
import numpy as np
import pytest

import tos_b200 as T
from test_band_sweep_gpu import forests
from test_diag_blocks_gpu import check
from test_gap_sweep_gpu import catalog, thinned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_px", [1, 2, 31, 32, 33, 63, 127, 128, 129])
@pytest.mark.parametrize("grid", [("[0:200]*50", "[0:1]*20"), ("[0:150]*150", "[0:1]*100"), ("[20:160]*35", "[0.2:0.9]*14")])
def test_lengths(engine, n_px, grid):
    los, px = forests(8, n_px, 0.71)
    check(engine, los, px, T.Grid.polar(*grid), 3586.0)


@pytest.mark.parametrize("short", [1, 15, 16, 17, 33, 64, 65, 128])
def test_short_beside_long(engine, short):
    """Every pair of two lengths: blocks with a long sightline, pair by pair without."""
    los, px = catalog([np.arange(5 * s, 5 * s + (200 if s % 2 else short)) for s in range(9)])
    check(engine, los, px, T.Grid.polar(), 3586.0)


@pytest.mark.parametrize("grid", [("[0:120]*120", "[0:1]*60"), ("[0:150]*25", "[0:1]*4")])
def test_masked_and_unlike(engine, grid):
    rng = np.random.default_rng(23)
    los, px = catalog([thinned(rng, 9 * s, 400, 300) for s in range(9)])
    check(engine, los, px, T.Grid.polar(*grid), 3586.0)
    los, px = forests(9, 260, 0.7)
    for s in range(9):  # every sightline its own step
        px["distance"][260 * s:260 * (s + 1)] = 3800 + 3 * s + (0.55 + 0.04 * s) * np.arange(260)
    check(engine, los, px, T.Grid.polar(*grid), 3586.0)


def test_empty_and_groups(engine):
    los, px = catalog([np.arange(4 * s, 4 * s + n) for s, n in enumerate([40, 1, 60, 0, 90, 128, 3, 0, 64])])
    los["group"] = np.arange(9) % 2
    g = T.Grid.polar()
    cat = T.Catalog(engine, los, px, 6)
    bins, rows, st = T.xi_run(engine, cat, g, 3586.0, per_group=True)
    exact, erows, _ = T.xi_run(engine, cat, g, 3586.0, per_group=True, exact=True)
    cat.close()
    assert st["num_diag_items"] > 0 and bins["num_pairs"].sum() > 0
    assert np.array_equal(rows["num_pairs"], erows["num_pairs"])
    np.testing.assert_allclose(bins["wgt"], exact["wgt"], rtol=1e-9)
