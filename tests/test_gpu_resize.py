"""Image resize where a warp's rows, columns and taps end: images of three pixels to some
hundred a side, scales from a twentieth (twenty taps a row, no registers for them) over the
pyramid's to four, values of both signs.  Against the oracle, bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import geye_gb300 as g
    with g.Context(0) as c:
        yield c


@pytest.mark.parametrize("scale", [0.05, 0.26, 0.34, 0.49, 0.5, 0.5359, 0.7071, 0.933, 0.999, 1.001, 1.6, 4.0])
@pytest.mark.parametrize("h,w", [(3, 3), (31, 8), (32, 9), (33, 64), (65, 7), (96, 250), (241, 131)])
def test_resize(ctx, h, w, scale):
    rng = np.random.default_rng([h, w])
    img = np.ascontiguousarray(rng.normal(0, 100, (3, w, h)), np.float32)
    if int(np.float32(h) * np.float32(scale) + 0.5) < 1 or int(np.float32(w) * np.float32(scale) + 0.5) < 1:
        pytest.skip("empty result")
    got, want = ctx.resize(img, scale), O.resize(img, scale)
    assert got.shape == want.shape
    assert np.array_equal(got.view(np.int32), np.ascontiguousarray(want).view(np.int32))
