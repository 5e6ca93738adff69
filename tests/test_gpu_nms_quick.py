"""The quicksort's order inside the pipeline NMS: frames with equal scores over
large areas (every box, half of them, a few), at box counts on both sides of the
sizes where the sort changes hands (a block's shared memory, a block, the
cluster) and where the walk is cut in two; in both orders, as a frame's graph and
as a lane of a batch.  Kept records equal to the oracle's, bit for bit."""
import numpy as np
import pytest

from geye_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# (w, h): 1100 to 4700 boxes of the car model (one segment of shared memory, then two), 16 000 to 40 000
# (one for a block, then the cluster's first split), 157 000 and 242 000 (the walk of the person model is cut in two)
SIZES = [(200, 150), (320, 240), (431, 323), (640, 480), (1280, 720)]


def _frame(w, h, kind):
    f = synth.make_frame(w, h, seed=3)
    if kind == "flat":
        f[:] = 90
    elif kind == "half":
        f[:, w // 2:] = 90
    elif kind == "stripes":   # (period of a cell: runs of equal scores between other ones)
        f[:, (np.arange(w) // 8) % 2 == 0] = 140
    return f


def _same(got, want, where):
    assert got["num"] == want["K"], where
    for k in ("point", "or_point", "type"):
        assert np.array_equal(got[k], want[k]), (where, k)
    assert np.array_equal(got["score"].view(np.int32), want["score"].view(np.int32)), where


@pytest.fixture(scope="module")
def paths(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("nms_quick"))
    return [synth.write_model_csv(s, d) for s in (synth.CAR_SPEC, synth.PERSON_SPEC)]


@pytest.mark.parametrize("kind", ["flat", "half", "stripes", "rects"])
@pytest.mark.parametrize("w,h", SIZES)
def test_both_orders(paths, w, h, kind):
    import geye_gb300 as g
    frame = _frame(w, h, kind)
    want = [O.car_detection(O.Model(*p), frame, -0.5, 0.5) for p in paths]
    for order in (g.NMS_ORDER_KEY, g.NMS_ORDER_QUICKSORT):
        with g.Context(0) as c:
            c.set_nms_order(order)
            ms = [g.Model(c, *p) for p in paths]
            for _ in range(2):   # (the second one through the captured graph again)
                for m, (x, y) in enumerate(zip(c.detect_multi(frame, ms, -0.5, 0.5), want)):
                    _same(x, y, (order, m))
            for m in ms:
                m.close()


def test_batch_lanes(paths):
    import geye_gb300 as g
    frames = [_frame(w, h, k) for (w, h) in SIZES[1:4] for k in ("flat", "half", "rects")] + [_frame(1280, 720, "rects")]
    with g.Context(0, conv=g.CONV_BF16) as c:
        ms = [g.Model(c, *p) for p in paths]
        want = [c.detect_multi(f, ms, -0.5, 0.5) for f in frames]
        b = g.Batch(ms, conv=g.CONV_BF16, max_frames=len(frames))
        for _ in range(2):
            for i, (got, w) in enumerate(zip(b.run(frames, -0.5, 0.5), want)):
                for x, y in zip(got, w):
                    assert x["num"] == y["num"], i
                    for k in ("point", "or_point", "type"):
                        assert np.array_equal(x[k], y[k]), (i, k)
                    assert np.array_equal(x["score"].view(np.int32), y["score"].view(np.int32)), i
        b.close()
        for m in ms:
            m.close()
