"""Results and stage outputs through the buffers a context keeps between calls: more kept boxes
than the pinned block holds, arrays that outlive later calls and their context,
and the asynchronous paths on frames that change from call to call."""
import numpy as np
import pytest

from geye_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def paths(tmp_path_factory):
    return synth.write_model_csv(synth.CAR_SPEC, str(tmp_path_factory.mktemp("host_results")))


def _same(a, b):
    assert a["num"] == b["num"]
    for k in ("point", "or_point", "type", "scale", "score"):
        assert np.array_equal(a[k], b[k]), k


def test_more_kept_boxes_than_the_pinned_block(paths):
    import geye_gb300 as g
    frame = synth.make_frame(560, 420, seed=2)
    want = O.car_detection(O.Model(*paths), frame, -0.5, 0.99)
    with g.Context(0) as c:
        m = g.Model(c, *paths)
        got = c.car_detection(frame, m, -0.5, None, 0.99)
        c.detect_submit(frame, [m], -0.5, 0.99)
        late = c.detect_collect()[0]
        m.close()
    assert got["num"] == want["K"] > 2048
    assert np.array_equal(got["point"], want["point"]) and np.array_equal(got["score"].view(np.int32), want["score"].view(np.int32))
    _same(got, late)


def test_stage_arrays_outlive_calls_and_context(paths):
    import geye_gb300 as g
    frames = [synth.make_frame(333, 251, seed=s) for s in (1, 2)]
    c = g.Context(0)
    m = g.Model(c, *paths)
    first = c.calc_f_pyramid(frames[0], m)
    second = c.calc_f_pyramid(frames[1], m)
    boxes = c.get_boxes(*[first[0], first[2], first[1]], m, -0.5)
    again = c.calc_f_pyramid(frames[0], m)
    m.close()
    c.close()
    assert any(not np.array_equal(a, b) for a, b in zip(first[0], second[0]))
    for a, b in zip(first[0], again[0]):
        assert np.array_equal(a.view(np.int32), b.view(np.int32))
    om = O.Model(*paths)
    P = O.Pyramid(om, frames[0])
    for l, f in enumerate(first[0]):
        assert np.array_equal(f.view(np.int32), P.feat(l).view(np.int32)), l
    assert boxes.shape[0] > 0 and np.isfinite(boxes).all()


def test_frames_change_from_call_to_call(paths):
    import geye_gb300 as g
    frames = [synth.make_frame(320, 240, seed=s) for s in range(5)]
    blank = np.zeros((240, 320, 3), np.uint8)
    with g.Context(0) as c:
        m = g.Model(c, *paths)
        want = [c.detect_multi(f, [m], 0.4, 0.5)[0] for f in frames]
        none = c.detect_multi(blank, [m], 5.0, 0.5)[0]
        assert none["num"] == 0
        with g.Server([m], conv=g.CONV_FP32, max_slots=2, thresh=0.4) as srv:
            tickets = [srv.submit(k % 3, f) for k, f in enumerate(frames * 2)]   # (more than the slots: some wait)
            srv.drain()
            got = {d["ticket"]: d["results"][0] for d in srv.poll(64)}
        for k, t in enumerate(tickets):
            _same(got[t], want[k % 5])
        b = g.Batch([m], conv=g.CONV_FP32, max_frames=3)
        for shift in range(2):
            for k, r in enumerate(b.run(frames[shift:shift + 3], 0.4, 0.5)):
                _same(r[0], want[shift + k])
        b.close()
        m.close()
