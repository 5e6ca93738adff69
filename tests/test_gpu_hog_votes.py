"""HOG votes read four pixels at a time: images whose blocks end at every remainder of four
pixels, every bin size, bin sizes whose pixel columns are not a multiple of four
long (a model of four-pixel bins has levels of two), flat and saturated areas.
Against the oracle, bit for bit."""
import dataclasses

import numpy as np
import pytest

from geye_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import geye_gb300 as g
    with g.Context(0) as c:
        yield c


@pytest.mark.parametrize("sbin", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("h,w", [(24, 24), (25, 27), (30, 41), (67, 45), (94, 131), (119, 90)])
def test_features(ctx, h, w, sbin):
    img = synth.make_frame(w, h, seed=h)[:, :, ::-1].astype(np.float32)
    img[: h // 4] = 0
    img[:, : w // 5] = 255
    img = np.ascontiguousarray(img.transpose(2, 1, 0))
    got, want = ctx.calc_feature(img, sbin), O.calc_feature(img, sbin)
    assert np.array_equal(np.ascontiguousarray(got).view(np.int32), np.ascontiguousarray(want).view(np.int32))


@pytest.mark.parametrize("w,h", [(163, 121), (202, 150), (187, 147)])
def test_frame_of_small_bins(ctx, tmp_path, w, h):
    import geye_gb300 as g
    spec = dataclasses.replace(synth.CAR_SPEC, name="car4", sbin=4)
    paths = synth.write_model_csv(spec, str(tmp_path))
    frame = synth.make_frame(w, h, seed=w)
    m = g.Model(ctx, *paths)
    got = ctx.car_detection(frame, m, -0.5, None, 0.5)
    m.close()
    want = O.car_detection(O.Model(*paths), frame, -0.5, 0.5)
    assert got["num"] == want["K"] > 0
    assert np.array_equal(got["point"], want["point"])
    assert np.array_equal(got["score"].view(np.int32), want["score"].view(np.int32))
