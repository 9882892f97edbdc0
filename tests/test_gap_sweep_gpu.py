"""GPU parity of the band sweep over sightlines with gaps at the sizes where it
can go wrong: at the limits of which sightlines it takes, mixed with contiguous
ones, spans beyond the shared-memory staging, runs of missing pixels longer than
a warp's steps, stretches of zero weight, and loglam values that are not a
function of the distance grid.  Counts equal the FP64 oracle's; sums agree to
the suite's REL_TOL (exactly zero where every term is zero)."""
import numpy as np
import pytest

import tos_b200 as T
from helpers import assert_counts_equal, assert_sums_close
from oracle import oracle

pytestmark = pytest.mark.gpu

GRIDS = {
    "cartesian": lambda: T.Grid.cartesian("[0:120]*30", "[0:60]*29"),
    "one_band": lambda: T.Grid.cartesian("[0:200]*1", "[0:60]*3"),
    "min_first": lambda: T.Grid.cartesian("[12:120]*27", "[0:60]*11"),
    "min_offset": lambda: T.Grid.cartesian("[10:120]*40", "[5:60]*11"),
    "observing": lambda: T.Grid.observing("[0:0.01]*33"),
}


def check(engine, los, px, g, scale=3586.0):
    cat = T.Catalog(engine, los, px, 6)
    bins, _, st = T.xi_run(engine, cat, g, scale)
    cat.close()
    ref = oracle.xi(los, px, 6, g.type, g.axes_array(), scale, mode=1)[0]
    ref_abs = oracle.xi(los, px, 6, g.type, g.axes_array(), scale, mode=2)[0]
    assert_counts_equal(bins, ref)
    assert_sums_close(bins, ref, ref_abs)
    return bins, st


def catalog(kept, seed=5, step=0.75):
    """Sightlines whose pixels are the grid values `kept[s]` (indices)."""
    rng = np.random.default_rng(seed)
    los = np.zeros(len(kept), dtype=T.SIGHTLINE_DTYPE)
    n = [len(k) for k in kept]
    px = np.zeros(sum(n), dtype=T.PIXEL_DTYPE)
    for s, k in enumerate(kept):
        los[s]["ra"], los[s]["dec"] = 3.0 + 2e-3 * s, 0.3 + 1.5e-3 * (s % 3)
        los[s]["pixel_offset"], los[s]["num_pixels"] = sum(n[:s]), n[s]
        p = px[sum(n[:s]):sum(n[:s + 1])]
        p["distance"] = 3800.0 + step * k
        p["loglam"] = 3.6 + 2e-5 * k
        p["value"] = rng.normal(0, 0.2, n[s])
        p["weight"] = rng.uniform(0.5, 2, n[s])
    return los, px


def thinned(rng, first, span, n):
    """n of `span` consecutive values, the first and the last among them."""
    inner = rng.choice(np.arange(1, span - 1), n - 2, replace=False) if n > 2 else np.zeros(0, int)
    return first + np.sort(np.concatenate([[0], inner, [span - 1]]).astype(int))


@pytest.mark.parametrize("grid", list(GRIDS))
def test_mixed_sightlines(engine, grid):
    """Contiguous, masked in windows, sparse, short and one-pixel sightlines."""
    rng = np.random.default_rng(11)
    kept = [np.arange(0, 400)]
    kept += [thinned(rng, 13 * s, 350, 300) for s in range(4)]
    kept += [np.concatenate([np.arange(0, 90), np.arange(290, 360)]) + 31 * s for s in range(4)]
    kept += [thinned(rng, 50, span, n) for n, span in ((47, 48), (48, 49), (48, 144), (48, 145), (100, 300))]
    kept += [np.array([77]), np.array([5, 390]), np.arange(100, 148), np.arange(200, 201)]
    los, px = catalog(kept)
    bins, st = check(engine, los, px, GRIDS[grid]())
    assert bins["num_pairs"].sum() > 0
    if grid == "min_offset":  # bins of equal pixels within FP32 of a bin edge: no sweep
        assert st["num_run_items"] == 0
    else:
        assert st["num_grid_items"] < st["num_run_items"] == st["num_sightline_pairs_used"]


@pytest.mark.parametrize("span", [1, 2, 31, 32, 33, 63])
def test_missing_runs(engine, span):
    """One gap of `span` values in every sightline, at every phase of a row step."""
    kept = [np.concatenate([np.arange(0, 40 + s), np.arange(40 + s + span, 120)]) for s in range(9)]
    los, px = catalog(kept)
    check(engine, los, px, GRIDS["cartesian"]())


@pytest.mark.parametrize("span", [1600, 2600])
def test_long_spans(engine, span):
    rng = np.random.default_rng(span)
    kept = [thinned(rng, 9 * s, span, span * 2 // 3) for s in range(4)]
    los, px = catalog(kept, step=0.125)
    _, st = check(engine, los, px, GRIDS["cartesian"]())
    assert st["num_grid_items"] == 0 and st["num_run_items"] == 6


def test_zero_weight_stretches(engine):
    rng = np.random.default_rng(17)
    los, px = catalog([thinned(rng, 5 * s, 300, 250) for s in range(12)])
    for s in range(len(los)):
        o = int(los[s]["pixel_offset"])
        a = int(rng.integers(0, 230))
        px[o:o + a]["weight"] = 0
        px[o + a + 20:o + 250]["weight"] = 0
    bins, _ = check(engine, los, px, T.Grid.cartesian("[0:200]*100", "[0:60]*50"))
    assert np.any((bins["num_pairs"] > 0) & (bins["wgt"] == 0)) and np.any(bins["wgt"] > 0)


@pytest.mark.parametrize("gaps", [False, True])
def test_loglam_of_each_pixel(engine, gaps):
    """Loglam not a function of the distance: every sightline its own offset."""
    rng = np.random.default_rng(19)
    los, px = catalog([thinned(rng, 5 * s, 200, 160) if gaps else np.arange(5 * s, 5 * s + 160) for s in range(10)])
    for s in range(len(los)):
        px["loglam"][160 * s:160 * (s + 1)] += np.float32(1e-3 * s)
    _, st = check(engine, los, px, GRIDS["cartesian"]())
    assert st["num_grid_items"] == 0 and st["num_run_items"] == st["num_sightline_pairs_used"] > 0
