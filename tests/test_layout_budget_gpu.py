"""A masked catalogue's layout on the common grid is optional: a server whose
budget has no room for it takes the catalogue without it, whether or not an
earlier run built it, and the counts are the FP64 oracle's either way; once the
catalogue is detached its runs build the layout again."""
import numpy as np
import pytest

import tos_b200 as T
from helpers import assert_counts_equal, assert_sums_close
from oracle import oracle
from test_gap_sweep_gpu import catalog

pytestmark = pytest.mark.gpu

GRIDS = (T.Grid.cartesian("[0:120]*8", "[0:60]*9"), T.Grid.observing("[0:0.01]*9"))


def masked():
    rng = np.random.default_rng(3)
    kept = [np.arange(s, s + 900) for s in range(6)]
    kept += [s + np.sort(rng.choice(900, 800, replace=False)) for s in range(60)]
    return catalog(kept, step=0.25)


@pytest.fixture(scope="module")
def reference():
    los, px = masked()
    return [[oracle.xi(los, px, 6, g.type, g.axes_array(), 3586.0, mode=m)[0] for m in (1, 2)] for g in GRIDS]


def check(bins, ref):
    assert_counts_equal(bins, ref[0])
    assert_sums_close(bins, *ref)


@pytest.mark.parametrize("built_before", [False, True])
def test_attach_without_room(engine, reference, built_before):
    los, px = masked()
    with T.Server(0, slots=1, memory_budget_bytes=10**10) as srv:
        cat = T.Catalog(engine, los, px, 6)
        srv.attach(cat)
        full = srv.status()["resident_bytes"]
        srv.detach(cat)
        cat.close()
    cat = T.Catalog(engine, los, px, 6)
    bare = cat.device_bytes()
    layout = 2 * 64 * len(px)  # at least: both axes
    assert full - bare > layout
    if built_before:
        for g, ref in zip(GRIDS, reference):
            check(T.xi_run(engine, cat, g, 3586.0)[0], ref)
        assert cat.device_bytes() > bare + layout
    budget = full - layout // 2 + (cat.device_bytes() - full if built_before else 0)
    with T.Server(0, slots=1, memory_budget_bytes=budget) as srv:
        srv.attach(cat)
        assert srv.status()["resident_bytes"] < budget - layout // 4
        for g, ref in zip(GRIDS, reference):
            bins, _, st, _ = srv.submit(cat, g, 3586.0).wait()
            check(bins, ref)
            assert 0 < st["num_grid_items"] < st["num_run_items"]
        without = cat.device_bytes()
        bins, _, _ = T.xi_run(engine, cat, GRIDS[0], 3586.0)  # attached: not built by a run of one's own either
        check(bins, reference[0])
        assert cat.device_bytes() - without < layout // 4
        srv.detach(cat)
    for g, ref in zip(GRIDS, reference):
        check(T.xi_run(engine, cat, g, 3586.0)[0], ref)
    assert cat.device_bytes() > bare + layout
    cat.close()
