"""Which kernel a brute-force count runs: points in lines of equal steps go as
lines, points just off that structure do not; and a tuned launch shape is used
only for the kernel it was measured on."""
import numpy as np
import pytest

import tos_b200 as T
from test_brute_lines_gpu import lines

pytestmark = pytest.mark.gpu


def run(engine, pts, nbins=30):
    out = T.brute_run(engine, pts, 0.0, 60.0, nbins)
    return out, T.brute_last_shape(engine)


@pytest.mark.parametrize("n_lines,length", [(32, 8), (33, 9), (95, 17), (32, 64), (32, 1024)])
def test_lines_run_as_lines(engine, n_lines, length):
    assert run(engine, lines(n_lines, length, step=(0, 0, 0.25)))[1][0] == length


@pytest.mark.parametrize("n_lines,length", [(31, 16), (40, 7), (32, 1025)])
def test_outside_the_limits(engine, n_lines, length):
    assert run(engine, lines(n_lines, length, step=(0, 0, 0.25)))[1][0] == 0


def test_off_the_structure(engine):
    off = lines(40, 16, seed=5)
    off[333, 1] += 0.25
    inexact = lines(40, 16, seed=7)
    inexact[:, :3] *= np.float32(0.1)
    for pts in (off, lines(40, 16, seed=6)[:-3], inexact):
        assert run(engine, pts)[1][0] == 0


@pytest.mark.parametrize("side", [24, 60])  # 131,072 points are no whole number of lines of 60
def test_pick_is_of_its_own_kernel(side):
    rng = np.random.default_rng(1)
    grid = T.synth.grf_grid(side, 4.0 * side, seed=9)
    scattered = np.concatenate([rng.uniform(0, 80, (5000, 3)), rng.normal(size=(5000, 2))], 1).astype(np.float32)
    with T.Engine(0) as eng:
        before, default = run(eng, scattered)
        assert default[0] == 0
        k, w = T.brute_tune(eng, grid, 0.0, 60.0, 30)
        assert T.brute_last_shape(eng)[0] == side and k == 1
        assert run(eng, grid)[1] == (side, 1, w)
        after, shape = run(eng, scattered)
        assert shape == default  # not the grid's pick
        k2, w2 = T.brute_tune(eng, scattered, 0.0, 60.0, 30)
        assert run(eng, scattered)[1] == (0, k2, w2)
        assert run(eng, grid)[1] == (side, 1, w)
        for a, b in zip(before[:3], after[:3]):
            assert np.array_equal(a, b)
