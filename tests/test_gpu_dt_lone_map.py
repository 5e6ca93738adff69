"""Plans with a single part map: one component of one part and one kept level.  Its distance transform
starts from a cleared count of left-over strips at every launch: on a new plan, when a frame is run
again and when the strip size is tuned; maps that read their own range and larger ones, windows of the
strips and of the general form in either direction.  Against the oracle, bit for bit."""
import numpy as np
import pytest

from geye_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# deformation weights (ax, bx, ay, by): windows of the strips; wider than theirs along y, along x, along both
DEFS = {"strips": ((0.02, 0.05), (0.0, 0.01), (0.02, 0.05), (0.0, 0.01)),
        "wide_y": ((0.02, 0.05), (0.0, 0.01), (1e-5, 1e-5), (0.0, 0.0)),
        "wide_x": ((1e-5, 1e-5), (0.0, 0.0), (0.02, 0.05), (0.0, 0.01)),
        "wide": ((1e-5, 1e-5), (0.0, 0.0), (1e-5, 1e-5), (0.0, 0.0))}


def _paths(tmp_path, root, kind):
    spec = synth.ModelSpec(f"lone_{kind}", roots=[root], seed=5, parts=[[(6, 6)]], offsets=[0.1], def_ranges=DEFS[kind])
    return synth.write_model_csv(spec, str(tmp_path))


@pytest.mark.parametrize("kind", sorted(DEFS))
@pytest.mark.parametrize("w,h", [(144, 96), (431, 323), (900, 700)])   # part maps of 600, 7600 and 36 000 values
def test_get_boxes_of_one_level(tmp_path, w, h, kind):
    import geye_gb300 as g
    paths = _paths(tmp_path, (6, 8), kind)
    om = O.Model(*paths)
    n = om.m.interval + 1
    P = O.Pyramid(om, synth.make_frame(w, h, seed=7))
    full = P._p.contents.LEN
    P._p.contents.LEN = n   # the first octave and one level above it
    S = O.Scores(om, P)
    want, _ = S.boxes(-0.5)
    feats = [P.feat(l) for l in range(n)]
    with g.Context(0) as c:
        m = g.Model(c, *paths)
        for _ in range(3):
            got = c.get_boxes(feats, P.scales[:n], np.array(P.ftsize[:n]), m, -0.5)
            assert got.shape == want.shape and want.shape[0] > 0
            assert np.array_equal(got.view(np.int32), want.view(np.int32))
        m.close()
    P._p.contents.LEN = full


@pytest.mark.parametrize("kind", sorted(DEFS))
@pytest.mark.parametrize("graphs", [True, False])
def test_frames_of_one_level(tmp_path, monkeypatch, kind, graphs):
    import geye_gb300 as g
    if not graphs:
        monkeypatch.setenv("GEYE_NO_GRAPHS", "1")
    paths = _paths(tmp_path, (10, 18), kind)
    w, h = 160, 96   # ten by eighteen cells: the root fits at one level
    frames = [synth.make_frame(w, h, seed=s) for s in (1, 2)]
    om = O.Model(*paths)
    want = [O.car_detection(om, f, -9.0, 0.5) for f in frames]
    P = O.Pyramid(om, frames[0])
    assert sum(not s for s in O.Scores(om, P).skipped[om.m.interval:]) == 1
    with g.Context(0) as c:
        m = g.Model(c, *paths)
        for k in range(6):   # (the strip size is tuned after the first)
            got, w_ = c.detect_multi(frames[k % 2], [m], -9.0, 0.5)[0], want[k % 2]
            assert got["num"] == w_["K"]
            for f in ("point", "or_point", "type"):
                assert np.array_equal(got[f], w_[f]), f
            assert np.array_equal(got["score"].view(np.int32), w_["score"].view(np.int32))
            score = c.score_map(m, om.m.interval, 0)
            ref = O.Scores(om, O.Pyramid(om, frames[k % 2])).score(om.m.interval, 0)
            assert np.array_equal(score.view(np.int32), ref.view(np.int32))
        m.close()
