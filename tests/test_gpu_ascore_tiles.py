"""A_SCORE's tiles of 16 x 32 pixels, four of a column to a thread: frames that end at every
remainder of a quad and around a tile's edge, cells of two to four pixels (three of them in a
quad), more maps than are staged at a time.  Against the oracle, bit for bit."""
import dataclasses

import numpy as np
import pytest

from geye_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,sbin,interval", [
    (176, 128, 8, 10), (177, 129, 8, 10), (191, 130, 8, 10), (192, 131, 8, 10), (193, 159, 8, 10), (225, 160, 8, 10),
    (163, 121, 4, 10), (202, 150, 4, 10), (187, 147, 8, 60)])
def test_tiles(tmp_path, w, h, sbin, interval):
    import geye_gb300 as g
    spec = dataclasses.replace(synth.CAR_SPEC, name="m", sbin=sbin, interval=interval)
    paths = synth.write_model_csv(spec, str(tmp_path))
    frame = synth.make_frame(w, h, seed=w)
    want_a = np.zeros((w, h), np.float32)
    want_a[::3, ::5] = 0.25
    got_a = want_a.copy()
    with g.Context(0) as ctx:
        m = g.Model(ctx, *paths)
        got = ctx.car_detection(frame, m, -0.5, got_a, 0.5)
        m.close()
    want = O.car_detection(O.Model(*paths), frame, -0.5, 0.5, a_score=want_a)
    assert got["num"] == want["K"]
    assert want_a.max() > 0
    assert np.array_equal(got_a.view(np.int32), want_a.view(np.int32))
