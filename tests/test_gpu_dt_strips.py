"""The distance transform at the edges of its strips, window sizes and general form: maps of
one to 1100 lines, value ranges and deformation weights that give windows from three to
beyond the strips' largest, weights that bound no window, infinite values.  Values and
displacements against the oracle's, bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import geye_gb300 as g
    with g.Context(0) as c:
        yield c


def _check(ctx, v, w):
    got, want = ctx.dt(v, *w), O.dt(v, *w)
    for k, (x, y) in enumerate(zip(got, want)):
        x, y = np.ascontiguousarray(x), np.ascontiguousarray(y)
        assert np.array_equal(x.view(np.int32), y.view(np.int32)), k


def _map(d0, d1, scale, seed=0):
    rng = np.random.default_rng([d0, d1, seed])
    return np.ascontiguousarray(scale * rng.normal(0, 1, (d1, d0)), np.float32)


# a strip has 8 to 64 rows: maps of one strip, of several, with a last strip of one row, with more columns than a stage
@pytest.mark.parametrize("d0,d1", [(1, 1), (1, 40), (40, 1), (2, 3), (7, 9), (8, 128), (9, 130), (17, 1100), (33, 65),
                                   (64, 16), (65, 17), (97, 140), (113, 151), (1100, 5), (300, 421)])
def test_sizes(ctx, d0, d1):
    _check(ctx, _map(d0, d1, 0.1), (0.03, 0.01, 0.05, -0.02))


# windows of about 3, 4, 5, 6, 8, 12, 16 (the strips' largest), 20, 40, 70 and the whole line, in each direction
@pytest.mark.parametrize("ay", [0.4, 0.05, 0.02, 0.004, 0.0015, 0.0005, 0.0001])
@pytest.mark.parametrize("ax", [0.4, 0.05, 0.02, 0.004, 0.0015, 0.0005, 0.0001])
def test_windows(ctx, ax, ay):
    _check(ctx, _map(75, 90, 0.1, 1), (ax, 0.1 * ax, ay, -0.2 * ay))


@pytest.mark.parametrize("w", [(0.0, 0.01, 0.05, 0.0), (0.05, 0.0, 0.0, -0.01), (-0.01, 0.0, 0.05, 0.0), (0.0, 0.0, 0.0, 0.0),
                               (1e-9, 0.0, 1e-9, 0.0), (0.01, 0.3, 0.01, -0.4)])
def test_weights_without_a_window(ctx, w):
    _check(ctx, _map(61, 47, 0.1, 2), w)


@pytest.mark.parametrize("scale", [1e-30, 1e-6, 30.0, 1e6])
def test_value_ranges(ctx, scale):
    _check(ctx, _map(70, 66, scale, 3), (0.03, 0.01, 0.05, -0.02))
    v = np.full((66, 70), np.float32(scale), np.float32)   # one value: every tie to the smaller index
    _check(ctx, v, (0.03, 0.01, 0.05, -0.02))
    _check(ctx, np.zeros((66, 70), np.float32) * np.float32(-1), (0.03, 0.01, 0.05, -0.02))


def test_infinite_values(ctx):
    v = _map(70, 66, 0.1, 4)
    v[3:9, 20:50] = np.inf
    _check(ctx, v, (0.03, 0.01, 0.05, -0.02))
