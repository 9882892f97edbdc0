"""GPU parity of the Polar diagonal sweep at the sizes where it can go wrong:
sightlines around its 16-row blocks and 64-diagonal groups, longer than the
shared-memory staging takes, of different lengths, and with masked pixels
(distances that jump inside a block); fine grids, whose blocks seldom hold one
key.  Counts equal the FP64 oracle's; sums agree to the suite's REL_TOL."""
import numpy as np
import pytest

import tos_b200 as T
from helpers import assert_counts_equal, assert_sums_close, small_catalog
from oracle import oracle
from test_band_sweep_gpu import forests
from test_xi_gpu import drop_pixels

pytestmark = pytest.mark.gpu


def check(engine, los, px, g, scale):
    cat = T.Catalog(engine, los, px, 6)
    bins, _, st = T.xi_run(engine, cat, g, scale)
    cat.close()
    ref = oracle.xi(los, px, 6, g.type, g.axes_array(), scale, mode=1)[0]
    ref_abs = oracle.xi(los, px, 6, g.type, g.axes_array(), scale, mode=2)[0]
    assert st["num_diag_items"] == st["num_sightline_pairs_used"] > 0
    assert bins["num_pairs"].sum() > 0
    assert_counts_equal(bins, ref)
    assert_sums_close(bins, ref, ref_abs)


@pytest.mark.parametrize("n_px", [1, 2, 15, 16, 17, 33, 64, 65, 127, 129])
def test_block_edges(engine, n_px):
    los, px = forests(7, n_px, 0.71)
    check(engine, los, px, T.Grid.polar(), 3586.0)


def test_uneven_lengths(engine):
    los, px = forests(8, 300, 0.66)
    for s, n in enumerate([300, 1, 299, 16, 80, 3, 150, 257]):
        los[s]["num_pixels"] = n
    check(engine, los, px, T.Grid.polar("[0:150]*37", "[0:1]*11"), 3586.0)


@pytest.mark.parametrize("n_px", [2600, 2900])
def test_long_sightlines(engine, n_px):
    los, px = forests(3, n_px, 0.0625)
    check(engine, los, px, T.Grid.polar("[0:120]*30", "[0:1]*20"), 3586.0)


@pytest.mark.parametrize("grid", [("[0:200]*50", "[0:1]*20"), ("[0:180]*400", "[0:1]*300"), ("[20:160]*35", "[0.2:0.9]*14")])
def test_masked_and_fine(engine, grid):
    los, px, meta = small_catalog(n=50, seed=31, size_deg=1.5, max_pixels=260)
    los, px = drop_pixels(los, px, 0.15, seed=9)
    check(engine, los, px, T.Grid.polar(*grid), meta["scale"])
