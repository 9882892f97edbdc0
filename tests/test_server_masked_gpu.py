"""Masked catalogues in the request server: their sweep (the band sweep for gaps)
runs in chunks like the others, so a short request that arrives while a long one
sweeps finishes first.  Both results equal their lone runs."""
import time

import numpy as np
import pytest

import tos_b200 as T
from test_server_gpu import GRIDS, assert_identical

pytestmark = pytest.mark.gpu


def mask(los, px, seed):
    """A window of 30 pixels missing from the middle of every forest."""
    rng = np.random.default_rng(seed)
    keep = np.ones(len(px), dtype=bool)
    first = los["pixel_offset"].astype(np.int64)
    at = first + rng.integers(5, 60, len(los))
    for k in range(30):
        keep[at + k] = False
    total = np.concatenate([[0], np.cumsum(keep)])
    out = los.copy()
    out["pixel_offset"] = total[first]
    out["num_pixels"] = total[first + los["num_pixels"]] - total[first]
    return out, px[keep]


def test_short_masked_request_overtakes_long_one(engine):
    los, px, meta = T.synth.full_survey(20000, seed=7, area_deg2=1250.0)
    big = T.Catalog(engine, *mask(los, px, 1), 6)
    los, px, s_meta = T.synth.small_patch(150, seed=21, size_deg=3.0)
    small = T.Catalog(engine, *mask(los, px, 2), 6)
    g = GRIDS["cartesian"]
    ref_big, _, st = T.xi_run(engine, big, g, meta["scale"])
    ref_small = T.xi_run(engine, small, g, s_meta["scale"])[0]
    assert st["num_grid_items"] == 0 and st["num_run_items"] == st["num_sightline_pairs_used"] > 2 * 131072
    try:
        with T.Server(0, slots=2, memory_budget_bytes=40 * 10**9) as srv:
            srv.set_policy("shortest", max_wait_s=30.0)
            srv.attach(big)
            srv.attach(small)
            rb = srv.submit(big, g, meta["scale"])
            time.sleep(0.05)
            rs = srv.submit(small, g, s_meta["scale"])
            bb, _, _, ib = rb.wait()
            bs, _, _, i_s = rs.wait()
    finally:
        big.close()
        small.close()
    assert_identical(bb, ref_big, "long request")
    assert_identical(bs, ref_small, "short request")
    assert i_s["start_s"] < ib["end_s"] and i_s["end_s"] < ib["end_s"]
