"""GPU parity of the grid (band) sweep at the sizes where it can go wrong:
bands around a warp's 31, sightlines of one pixel up to longer than the
shared-memory staging takes, stretches of zero weight, and loglam values that
are not a function of the distance grid.  Counts equal the FP64 oracle's;
sums agree to the suite's REL_TOL (exactly zero where every term is zero)."""
import numpy as np
import pytest

import tos_b200 as T
from helpers import assert_counts_equal, assert_sums_close, small_catalog
from oracle import oracle

pytestmark = pytest.mark.gpu


def check(engine, los, px, g, scale):
    cat = T.Catalog(engine, los, px, 6)
    bins, _, st = T.xi_run(engine, cat, g, scale)
    cat.close()
    ref = oracle.xi(los, px, 6, g.type, g.axes_array(), scale, mode=1)[0]
    ref_abs = oracle.xi(los, px, 6, g.type, g.axes_array(), scale, mode=2)[0]
    assert_counts_equal(bins, ref)
    assert_sums_close(bins, ref, ref_abs)
    return bins, st


@pytest.mark.parametrize("n0", [1, 15, 16, 31, 47])
@pytest.mark.parametrize("coord", ["cartesian", "observing"])
def test_band_counts(engine, coord, n0):
    los, px, meta = small_catalog(n=40, seed=41, size_deg=2.0)
    if coord == "cartesian":
        g = T.Grid.cartesian(f"[0:{4 * n0}]*{n0}", "[0:200]*37")
    else:
        g = T.Grid.observing(f"[0:{0.001 * n0}]*{n0}")
    bins, st = check(engine, los, px, g, meta["scale"])
    assert st["num_grid_items"] == st["num_sightline_pairs_used"] > 0
    assert bins["num_pairs"].sum() > 0


@pytest.mark.parametrize("max_pixels", [1, 2, 5, 33])
def test_short_sightlines(engine, max_pixels):
    los, px, meta = small_catalog(n=60, seed=42, size_deg=1.5, max_pixels=max_pixels)
    check(engine, los, px, T.Grid.cartesian("[0:120]*33", "[0:200]*50"), meta["scale"])


def forests(n_los, n_px, step, first=0, seed=3):
    """Sightlines of n_px consecutive pixels of one distance grid, at staggered starts."""
    rng = np.random.default_rng(seed)
    los = np.zeros(n_los, dtype=T.SIGHTLINE_DTYPE)
    px = np.zeros(n_los * n_px, dtype=T.PIXEL_DTYPE)
    for s in range(n_los):
        los[s]["ra"], los[s]["dec"] = 3.0 + 4e-3 * s, 0.3 + 3e-3 * (s % 3)
        los[s]["pixel_offset"], los[s]["num_pixels"] = s * n_px, n_px
        k = first + 7 * s + np.arange(n_px)
        p = px[s * n_px:(s + 1) * n_px]
        p["distance"] = 3800.0 + step * k
        p["loglam"] = 3.6 + 2e-5 * k
        p["value"] = rng.normal(0, 0.2, n_px)
        p["weight"] = rng.uniform(0.5, 2, n_px)
    return los, px


@pytest.mark.parametrize("n_px", [3399, 3400, 3401])
def test_long_sightlines(engine, n_px):
    los, px = forests(4, n_px, 0.0625)
    _, st = check(engine, los, px, T.Grid.cartesian("[0:100]*25", "[0:60]*29"), 3586.0)
    assert st["num_grid_items"] == 6


def test_zero_weight_stretches(engine):
    los, px, meta = small_catalog(n=30, seed=43, size_deg=1.5, max_pixels=250)
    rng = np.random.default_rng(6)
    for s in range(len(los)):  # most of each sightline without weight: bins whose every term is zero
        o, n = int(los[s]["pixel_offset"]), int(los[s]["num_pixels"])
        a = rng.integers(0, n - 20) if n > 20 else 0
        keep = px[o + a:o + a + 20].copy()
        px[o:o + n]["weight"] = 0
        px[o + a:o + a + 20] = keep
    bins, _ = check(engine, los, px, T.Grid.cartesian("[0:200]*100", "[0:200]*100"), meta["scale"])
    assert np.any((bins["num_pairs"] > 0) & (bins["wgt"] == 0)) and np.any(bins["wgt"] > 0)


def test_loglam_not_a_function_of_distance(engine):
    los, px = forests(6, 150, 0.75)
    o, n = int(los[2]["pixel_offset"]), int(los[2]["num_pixels"])
    px["loglam"][o:o + n] += np.float32(1e-3)
    _, st = check(engine, los, px, T.Grid.cartesian(), 3586.0)
    assert st["num_grid_items"] == 0 and st["num_run_items"] == 15
