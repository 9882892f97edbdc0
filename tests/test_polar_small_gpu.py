"""GPU parity of the Polar binning at small separations of unaligned pixels,
where the reference's float rounding of d1^2 (up to 2^-24 d1^2, about 1) cancels
against the transverse term: r^2 from 1e-6 to 10 at distances of 4,000 to 8,000.
Counts equal the FP64 oracle's, in the diagonal sweep (sorted sightlines) and in
the pixel-pair kernel (a sightline that is not)."""
import numpy as np
import pytest

import tos_b200 as T
from helpers import assert_counts_equal
from oracle import oracle

pytestmark = pytest.mark.gpu

DECADES = [1e-6, 1e-5, 1e-4, 1e-3, 1e-2, 1e-1, 1.0, 10.0]


def close_pairs(dist, theta, n_mu, first=None, per_decade=96, n=2000000):
    """Two sightlines `theta` apart whose p-th pixels have r^2 (as the reference
    computes it) spread over DECADES and mu just beyond the window around an
    edge of n_mu bins that is re-binned: (sightlines, pixels)."""
    rng = np.random.default_rng(n_mu)
    cos = np.cos(theta)

    def r_sq(d1, d2):
        return (d1 * d1).astype(np.float64) + (d2 - (np.float32(2) * d1).astype(np.float64) * cos) * d2

    d1 = np.unique((dist + rng.uniform(0, 0.2 * dist, n)).astype(np.float32))
    w = r_sq(d1, d1)  # what r^2 holds beside (d2 - d1)^2, up to 1e-4 of it
    d1 = np.concatenate([d1[(w > 0) & (w < 0.1)], rng.choice(d1, 2000, replace=False)])
    d2 = d1[:, None] + np.spacing(np.float32(dist)) * np.arange(1, 24, dtype=np.float32)
    d2 = np.concatenate([d2, d1[:, None] + rng.uniform(0, 2, (len(d1), 4))], 1).astype(np.float32).ravel()
    d1 = np.repeat(d1, 27)
    rsq = r_sq(d1, d2)
    t = np.abs(d2 - d1) / np.sqrt(np.maximum(rsq, 1e-30)) * n_mu
    window = 2.0 ** -min(13, 21 - int(n_mu + 2).bit_length())  # closer pairs are re-binned in FP64
    edge = np.abs(np.abs(t - np.round(t)) - 2 * window)
    pick = []
    for lo, hi in zip(DECADES, DECADES[1:]):
        k = np.nonzero((rsq > lo) & (rsq < hi) & (rsq >= (d2 - d1).astype(np.float64) ** 2))[0]
        pick.append(k[np.argsort(edge[k])[:per_decade]])
    pick = np.sort(np.concatenate(pick))
    d1, d2 = d1[pick], d2[pick]
    if first:
        d1, d2 = np.concatenate([[first[0]], d1]), np.concatenate([[first[1]], d2])
    order = np.argsort(d1, kind="stable")
    d1, d2 = d1[order], np.sort(d2)
    keep = np.concatenate([[True], (np.diff(d1) > 0) & (np.diff(d2) > 0)])
    d1, d2 = d1[keep], d2[keep]
    m = len(d1)
    los = np.zeros(2, dtype=T.SIGHTLINE_DTYPE)
    los["ra"], los["dec"] = 0.7, (0.0, theta)
    px = np.zeros(2 * m, dtype=T.PIXEL_DTYPE)
    px["distance"] = np.concatenate([d1, d2])
    px["loglam"] = np.tile(3.6 + 2e-5 * np.arange(m), 2)
    px["value"] = rng.normal(0, 0.2, 2 * m)
    px["weight"] = rng.uniform(0.5, 2, 2 * m)
    los["pixel_offset"], los["num_pixels"] = (0, m), m
    return los, px


# angles whose transverse term 2 (1 - c) d^2 lies within the rounding's range
@pytest.mark.parametrize("dist,rperp", [(4000.0, 0.3), (4757.0, 0.8991), (6100.0, 0.7), (8000.0, 1.3)])
@pytest.mark.parametrize("n_mu", [20, 50, 100, 300])
@pytest.mark.parametrize("is_sorted", [True, False])
def test_small_separations(engine, dist, rperp, n_mu, is_sorted):
    # one pair worked out by hand: r^2 = 1.24e-6, mu code 43 of 50
    first = (np.float32(4757.66064453125), np.float32(4757.66162109375)) if dist == 4757.0 else None
    theta = np.arccos(0.9999999821402769) if first else rperp / dist
    los, px = close_pairs(dist + 1 if first else dist, theta, n_mu, first=first)
    if not is_sorted:
        m = int(los["num_pixels"][0])
        px[:m] = px[:m][::-1]
    g = T.Grid.polar("[0:200]*50", f"[0:1]*{n_mu}")
    cat = T.Catalog(engine, los, px, 6)
    bins, _, st = T.xi_run(engine, cat, g, 3586.0)
    cat.close()
    ref = oracle.xi(los, px, 6, g.type, g.axes_array(), 3586.0, mode=1)[0]
    assert st["num_diag_items"] == (1 if is_sorted else 0) and st["num_sightline_pairs_used"] == 1
    assert bins["num_pairs"].sum() > 0
    assert_counts_equal(bins, ref)
