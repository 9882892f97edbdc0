"""A sweep whose barrier wait runs out (here: a limit of zero, so that the first
item's copy is never there in time) ends, reports it by name, and leaves the
engine usable: the same call with the default limit gives the right counts."""
import numpy as np
import pytest

import tos_b200 as T
from test_gap_sweep_gpu import catalog, check

pytestmark = pytest.mark.gpu

CASES = {
    "band": (lambda s: np.arange(9 * s, 9 * s + 300), lambda: T.Grid.cartesian("[0:120]*30", "[0:60]*29")),
    "band ": (lambda s: np.arange(9 * s, 9 * s + 60), lambda: T.Grid.observing("[0:0.01]*33")),  # short items
    "gap": (lambda s: np.delete(np.arange(9 * s, 9 * s + 300), [40, 41]), lambda: T.Grid.cartesian("[0:120]*30", "[0:60]*29")),
    "Polar": (lambda s: np.arange(9 * s, 9 * s + 300), lambda: T.Grid.polar()),
}


@pytest.mark.parametrize("name", list(CASES))
def test_wait_runs_out(name):
    kept, grid = CASES[name]
    los, px = catalog([kept(s) for s in range(8)])
    with T.Engine(0) as eng:
        with pytest.raises(T.TosError, match="INVALID_ARG"):
            eng.set_wait_limit(-1.0)
        eng.set_wait_limit(0.0)
        cat = T.Catalog(eng, los, px, 6)
        for _ in range(2):
            with pytest.raises(T.TosError, match=f"TIMEOUT: a wait of the {name.strip()} sweep"):
                T.xi_run(eng, cat, grid(), 3586.0)
        cat.close()
        eng.set_wait_limit(10.0)
        check(eng, los, px, grid())
