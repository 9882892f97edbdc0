"""TOS_XI_TUNE on catalogues whose pairs other sweeps take (short, masked and
uneven sightlines): the tuning run and the runs after it, of that catalogue and
of one whose dominant kernel is tuned, give the untuned results bit for bit."""
import numpy as np
import pytest

import tos_b200 as T
from test_gap_sweep_gpu import catalog

pytestmark = pytest.mark.gpu

KINDS = {
    "short": [np.arange(5 * s, 5 * s + 60) for s in range(20)],
    "masked": [np.delete(np.arange(5 * s, 5 * s + 300), [30, 31, 90]) for s in range(20)],
    "mixed": [np.arange(5 * s, 5 * s + (300 if s % 2 else 40)) for s in range(20)],
}


@pytest.mark.parametrize("grid", [T.Grid.cartesian("[0:120]*30", "[0:60]*29"), T.Grid.polar("[0:120]*80", "[0:1]*20"),
                                  T.Grid.observing("[0:0.01]*33")])
@pytest.mark.parametrize("kind", list(KINDS))
def test_tuning_other_sweeps(kind, grid):
    whole = catalog([np.arange(5 * s, 5 * s + 300) for s in range(20)])
    with T.Engine(0) as eng:
        cats = [T.Catalog(eng, *catalog(KINDS[kind]), 6), T.Catalog(eng, *whole, 6)]
        ref = [T.xi_run(eng, c, grid, 3586.0)[0] for c in cats]
        tuned = T.xi_run(eng, cats[0], grid, 3586.0, tune=True)[0]
        again = [T.xi_run(eng, c, grid, 3586.0)[0] for c in cats]
        last = T.xi_run(eng, cats[1], grid, 3586.0, tune=True)[0]
        for a, b in [(ref[0], tuned), (ref[0], again[0]), (ref[1], again[1]), (ref[1], last)]:
            assert a["num_pairs"].sum() > 0
            for f in a.dtype.names:
                assert np.array_equal(a[f], b[f])
        for c in cats:
            c.close()
