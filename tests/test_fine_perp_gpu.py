"""GPU parity of fine r_perp bins at small separations, where the reference's float
rounding of d1^2 cancels against the transverse term: bins of 1 down to 0.001 at
distances of 4,000 to 8,000, the grid at 0 and off it.  Counts equal the FP64
oracle's."""
import numpy as np
import pytest

import tos_b200 as T
from helpers import assert_counts_equal
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dist", [4000.0, 8000.0])
@pytest.mark.parametrize("perp", ["[0:50]*50", "[0:5]*50", "[0:4]*400", "[0.005:4.005]*400", "[0:2]*2000"])
def test_fine_perp(engine, dist, perp):
    rng = np.random.default_rng(int(dist))
    n = 700
    los = np.zeros(6, dtype=T.SIGHTLINE_DTYPE)
    los["ra"] = 0.7
    los["dec"] = np.cumsum([0, 0.2, 0.4, 0.7, 1.0, 1.4]) / dist
    los["pixel_offset"], los["num_pixels"] = n * np.arange(6), n
    px = np.zeros(6 * n, dtype=T.PIXEL_DTYPE)
    for s in range(6):
        p = px[n * s:n * (s + 1)]
        p["distance"] = np.sort(dist + rng.uniform(0, 60, n))
        p["loglam"] = 3.6 + 2e-5 * np.arange(n)
        p["value"], p["weight"] = rng.normal(0, 0.2, n), rng.uniform(0.5, 2, n)
    g = T.Grid.cartesian("[0:60]*10", perp)
    cat = T.Catalog(engine, los, px, 6)
    bins, _, st = T.xi_run(engine, cat, g, dist * 0.9)
    cat.close()
    ref = oracle.xi(los, px, 6, g.type, g.axes_array(), dist * 0.9, mode=1)[0]
    assert st["num_sightline_pairs_used"] > 0 and bins["num_pairs"].sum() > 1000
    assert_counts_equal(bins, ref)
