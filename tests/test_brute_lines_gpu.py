"""GPU parity of the brute-force count's two layouts at the sizes where they can
go wrong: points in lines of equal steps (line lengths around the offset
blocks, line counts around a warp's 32, skewed steps), points just off that
structure, coordinates whose FP32 differences are not exact, row-segment
remainders, and bins that take most of the pairs.  Counts equal the FP64
oracle's; weight sums agree to 1e-9 and signal sums, which cancel, to 1e-9 of
the sum of |terms|."""
import numpy as np
import pytest

import tos_b200 as T
from oracle import oracle

pytestmark = pytest.mark.gpu


def lines(n_lines, length, step=(0.0, 0.0, 4.0), spread=40.0, seed=1, quantum=0.25):
    rng = np.random.default_rng(seed)
    base = np.round(rng.uniform(0, spread, (n_lines, 1, 3)) / quantum) * quantum
    pos = base + np.arange(length)[None, :, None] * np.asarray(step)
    p = np.empty((n_lines * length, 5))
    p[:, :3] = pos.reshape(-1, 3)
    p[:, 3] = rng.normal(size=len(p))
    p[:, 4] = rng.uniform(0.5, 2, len(p))
    return p.astype(np.float32)


def check(engine, pts, rmin, rmax, nbins):
    ds, ws, ct, _ = T.brute_run(engine, pts, rmin, rmax, nbins)
    ods, ows, oct_ = oracle.brute(pts, rmin, rmax, nbins)
    assert np.array_equal(ct, oct_), np.nonzero(ct != oct_)[0][:10]
    np.testing.assert_allclose(ws, ows, rtol=1e-9)
    mag = np.abs(pts[:, 3] * pts[:, 4]).mean() ** 2 * np.maximum(oct_, 1)
    assert np.max(np.abs(ds - ods) / mag) < 1e-9
    again = T.brute_run(engine, pts, rmin, rmax, nbins)
    assert np.array_equal(ds, again[0]) and np.array_equal(ws, again[1])


@pytest.mark.parametrize("n_lines,length", [(32, 8), (33, 9), (64, 15), (40, 16), (31, 16), (95, 17), (32, 64)])
def test_lines(engine, n_lines, length):
    check(engine, lines(n_lines, length, seed=length), 0.0, 60.0, 30)


def test_skewed_steps_and_narrow_range(engine):
    check(engine, lines(50, 24, step=(0.5, -1.25, 2.0), seed=4), 5.0, 20.0, 61)


def test_one_point_off_its_line(engine):
    pts = lines(40, 16, seed=5)
    pts[333, 1] += 0.25
    check(engine, pts, 0.0, 60.0, 30)


def test_part_of_a_line_missing(engine):
    check(engine, lines(40, 16, seed=6)[:-3], 0.0, 60.0, 30)


def test_inexact_differences(engine):
    pts = lines(40, 16, seed=7)
    pts[:, :3] *= np.float32(0.1)
    check(engine, pts, 0.0, 6.0, 30)


@pytest.mark.parametrize("n", [2, 3, 32, 33, 34, 65, 1000, 2047, 2049])
def test_scattered_sizes(engine, n):
    rng = np.random.default_rng(n)
    pts = np.concatenate([rng.uniform(0, 80, (n, 3)), rng.normal(size=(n, 1)), rng.uniform(-1, 2, (n, 1))], 1)
    pts = pts.astype(np.float32)
    ds, ws, ct, _ = T.brute_run(engine, pts, 0.0, 70.0, 23)
    ods, ows, oct_ = oracle.brute(pts, 0.0, 70.0, 23)
    assert np.array_equal(ct, oct_)
    mag = 4.0 * np.maximum(oct_, 1)
    assert np.max(np.abs(ws - ows) / mag) < 1e-9 and np.max(np.abs(ds - ods) / mag) < 1e-9


@pytest.mark.parametrize("rmax,nbins", [(1.0, 3), (400.0, 1), (70.0, 300)])
def test_crowded_bins(engine, rmax, nbins):
    rng = np.random.default_rng(8)
    pts = np.concatenate([rng.uniform(0, 80, (4000, 3)), rng.normal(size=(4000, 1)),
                          rng.uniform(0.5, 2, (4000, 1))], 1).astype(np.float32)
    check(engine, pts, 0.0, rmax, nbins)
    check(engine, lines(64, 32, seed=9), 0.0, rmax, nbins)
